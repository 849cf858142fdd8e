// Host side of the standard quotient filter shared by its translation units
// (the layout kernels, the in-place updates and the cluster-local updates
// compile in parallel): geometry, scratch and the launchers.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <type_traits>

#include "host_common.cuh"
#include "sqf_build.cuh"
#include "sqf_extract.cuh"
#include "sqf_fallback.cuh"
#include "sqf_walk.cuh"

namespace gqf {

// ------------------------------------------------------------------ geometry
inline bool qr_ok(unsigned q, unsigned r)
{
    // quotientFilter.cu:46-47 asserts q + r <= 32 and (r + 3) % 8 == 0; a
    // 32-bit fingerprint would need `1 << 32` in the hash modulus (:268), so
    // q + r <= 31 here.  q >= 7 keeps a bucket at least 128 quotients.
    return (r + 3) % 8 == 0 && (r + 3) / 8 <= 2 && q >= 7 && q + r <= 31 && r >= 1;
}

struct SqfGeom {
    uint32_t q, r, bpe, nslots;
    size_t T;
};
inline SqfGeom geom_of(const gqf_sqf *qf)
{
    SqfGeom g;
    g.q = qf->qbits;
    g.r = qf->rbits;
    g.bpe = (g.r + 3) / 8;
    g.nslots = gqf_sqf_num_slots(g.q);
    g.T = gqf_sqf_table_bytes(g.q, g.r);
    return g;
}

inline uint32_t ceil_log2(uint64_t x)
{
    uint32_t l = 0;
    while ((1ull << l) < x) l++;
    return l;
}

struct LayoutPlan {
    BucketGeom g;
    uint32_t stride;     // speculative bucket stride (items)
    uint64_t n_expect;   // items it was made for
    uint32_t cap_items;  // per-CTA item capacity of k_bucket_layout
    size_t smem;
};

// Layout buckets of an in-place update: 8192 quotients (three CTAs per SM
// hold their sets, index and tile), fewer where the filter would otherwise
// give less than 512 buckets, down to 1024.
inline uint32_t update_tb(uint32_t q) { return std::min<uint32_t>(q, std::min<uint32_t>(13, std::max<uint32_t>(10, q > 9 ? q - 9 : 0))); }

template <typename K>
static cudaError_t set_smem(K kernel, size_t bytes)
{
    // the attribute is per function and device; set it only when it grows
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, size_t> done;
    const std::pair<const void *, int> key(reinterpret_cast<const void *>(kernel), current_device());
    std::lock_guard<std::mutex> lk(mu);
    size_t &cur = done[key];
    if (bytes <= cur) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) cur = bytes;
    return e;
}

// ------------------------------------------------------------ the pipeline
// Scratch for one rebuild: control words, look-back descriptors, fix-ups,
// the bucketed batch (B) and optionally the table's extracted contents (A).
struct Scratch {
    uint32_t *bcnt;              // nb  : batch items per bucket
    unsigned long long *status;  // nb  : look-back descriptors
    uint32_t *ticket;
    uint32_t *fix_cnt;
    uint32_t *a_dups;  // table holds duplicate fingerprints (set by extraction)
    uint32_t *fused_fail;  // the in-place update could not decode some bucket
    uint8_t *snap;         // table snapshot of the in-place update
    FallbackArgs fb;       // the rebuild behind a queued one
    uint32_t *bbase;  // nb+1: exact batch bases
    uint32_t *fix_list;
    uint32_t fix_cap;
    uint32_t *bitems;  // batch fingerprints
    void *rems;        // k_group_layout: remainders of large buckets
    // extracted table contents
    Counts3 *tiles;
    uint32_t *Q, *E, *abase, *acnt;
    uint32_t *E2, *a2base, *a2cnt;
    size_t ctrl_bytes;
};

struct ScratchReq {
    uint32_t nb;
    size_t batch_items;  // capacity of the bucketed batch
    bool extract;   // table contents needed
    bool extract2;  // second table (merge)
    uint32_t nslots;
    size_t snap_bytes = 0;  // in-place update: snapshot of the table
    uint32_t upd_nb = 0;    // and its layout buckets
    bool every_fix = false; // room for a fix-up of every quotient
    uint32_t rem_bytes = 0; // k_group_layout: scratch bytes per item
    const SqfGeom *fallback = nullptr;  // in-place update: the rebuild behind it
};

inline uint32_t fallback_buckets(uint32_t q) { return q > FB_TB ? 1u << (q - FB_TB) : 1u; }
// The rebuild's own buffers, apart from the lists (tiles, Q, E, E2, bitems)
// and the words that start at zero.
template <typename C>
void carve_fallback(C &c, FallbackArgs &f, const SqfGeom &tg, bool two)
{
    const uint32_t nb = fallback_buckets(tg.q);
    f.lay.status = c.template take<unsigned long long>(nb);
    f.lay.ticket = c.template take<uint32_t>(1, 4);
    f.lay.fix_cnt = c.template take<uint32_t>(1, 4);
    f.dups = c.template take<uint32_t>(1, 4);
    f.bcnt = c.template take<uint32_t>(nb);
    f.bfill = c.template take<uint32_t>(nb);
    f.bbase = c.template take<uint32_t>(nb);
    f.abase = c.template take<uint32_t>(nb);
    f.acnt = c.template take<uint32_t>(nb);
    if (two) f.b2cnt = c.template take<uint32_t>(nb);
}

inline Scratch carve(void *base, const ScratchReq &r, bool sizing_only, size_t *bytes_out)
{
    Scratch s{};
    auto lay = [&](auto &c) {
        size_t nb = r.nb;
        s.bcnt = c.template take<uint32_t>(nb, 8);
        s.status = c.template take<unsigned long long>(std::max<size_t>(nb, r.upd_nb), 8);
        s.ticket = c.template take<uint32_t>(1, 4);
        s.fix_cnt = c.template take<uint32_t>(1, 4);
        s.a_dups = c.template take<uint32_t>(1, 4);
        s.fused_fail = c.template take<uint32_t>(1, 4);
        s.fb.bar = c.template take<uint32_t>(4, 4);
        s.ctrl_bytes = c.off;
        s.bbase = c.template take<uint32_t>(nb + 1);
        s.fix_cap = std::max<uint32_t>(65536u, r.every_fix ? r.nslots : r.nslots / 8);
        s.fix_list = c.template take<uint32_t>(s.fix_cap);
        s.bitems = c.template take<uint32_t>(std::max<size_t>(r.batch_items, 1));
        s.rems = r.rem_bytes ? c.template take<uint8_t>((std::max<size_t>(r.batch_items, 1) +
                                                         (r.extract ? r.nslots : 0) + (r.extract2 ? r.nslots : 0)) *
                                                        r.rem_bytes)
                             : nullptr;
        if (r.extract) {
            size_t ntiles = (r.nslots + EXTRACT_TILE - 1) / EXTRACT_TILE;
            s.tiles = c.template take<Counts3>(ntiles + 1);
            s.Q = c.template take<uint32_t>(r.nslots);
            s.E = c.template take<uint32_t>(r.nslots);
            s.abase = c.template take<uint32_t>(nb + 1);
            s.acnt = c.template take<uint32_t>(nb);
            if (r.extract2) {
                s.E2 = c.template take<uint32_t>(r.nslots);
                s.a2base = c.template take<uint32_t>(nb + 1);
                s.a2cnt = c.template take<uint32_t>(nb);
            }
        }
        s.snap = r.snap_bytes ? c.template take<uint8_t>(r.snap_bytes) : nullptr;
        if (r.fallback) carve_fallback(c, s.fb, *r.fallback, r.extract2);
    };
    if (sizing_only) {
        Sizer z;
        lay(z);
        *bytes_out = z.off;
    } else {
        Carver c(base);
        lay(c);
        *bytes_out = c.off;
    }
    return s;
}

// Bucket layout of A and B into the table, fix-ups included (sqf_layout.cuh);
// with a gate, by the general kernel, if *gate is set.
template <int BPE>
int launch_layout(const LayoutPlan &p, const SqfGeom &tg, uint8_t *table, const BucketSrc &A, const BucketSrc &B,
                  int op, int nodup, bool set_ok, const uint32_t *a_dups, Scratch &sc, uint32_t *err, cudaStream_t s,
                  const uint32_t *gate = nullptr);
// In-place update of one-byte slots (sqf_inplace.cu).
int launch_update(const LayoutPlan &p, const SqfGeom &tg, uint8_t *table, const uint8_t *src2, const BucketSrc &B,
                  int op, Scratch &sc, uint32_t *err, cudaStream_t s);
// Slots an update walks before it gives the stretch up.  On a nearly full
// table the walks are lost time: the larger the table, the more its update as
// a whole costs, and the longer they may be.
inline uint32_t walk_limit(uint32_t q)
{
    return std::min(FAR_SLOTS, 1280u << (q > 22 ? std::min(q - 22, 2u) : 0));
}
// Cluster-local insert or delete (sqf_local.cu).  A synchronous call on
// one-byte slots that met a stretch too long to walk leaves the table as it
// was and sets *far; behind the others the rebuild runs on the device.
template <int BPE>
int local_update(const gqf_sqf *qf, const uint32_t *keys, uint32_t n, int op, cudaStream_t s, float *ms, bool *far);
void load_local_kernels();
void load_inplace_kernels();
size_t local_update_bytes(const SqfGeom &tg, uint32_t n, int op);
// The gated rebuild: gate, src, src2, snap, keys, n and the buffers are set.
// With `lists`, only the old contents' lists, in buckets of that geometry.
template <int BPE>
int launch_fallback(FallbackArgs &f, const SqfGeom &tg, uint8_t *table, int op, int nodup, uint32_t *err,
                    cudaStream_t s, const BucketGeom *lists = nullptr);

}  // namespace gqf

// An update done on the whole table by one cooperative launch, queued behind
// the update's own kernels and doing nothing unless they set its gate:
//   - a cluster-local update met a stretch too long to walk (sqf_update.cuh;
//     the table is then unchanged): one-byte tables are updated in place from
//     a snapshot, bucket by bucket, as k_set_update does;
//   - an in-place update, or that one, met a bucket it cannot decode (a table
//     holding duplicate fingerprints, a run past its slice): the old contents
//     are extracted, from the snapshot, and every bucket is laid out again
//     from both lists (as remainder sets where no copies are kept: any number
//     of items).
// One launch, because the usual case is the empty one: a kernel per step was
// 12 to 18 launches behind every queued in-place update or merge (q = 20, an
// insert of a key per 8 quotients: 117 us, now 67).
#pragma once

#include "grid_sync.cuh"
#include "sqf_build.cuh"
#include "sqf_extract.cuh"

namespace gqf {

constexpr int FB_THREADS = EXTRACT_THREADS;
constexpr uint32_t FB_TB = 13;  // quotients per bucket: 32 per thread (a smaller filter is one bucket)
static_assert((1u << FB_TB) == FB_THREADS * 32, "one layout CTA shape");
// Items a bucket of a table with copies, or of two-byte slots, may hold: what
// its u16 counters allow, eight times the average.
constexpr uint32_t FB_CAP = 65520;

struct FallbackArgs {
    const uint32_t *gate;  // run only if one of these bits is set in *gate
    uint32_t gate_bits;
    LayoutArgs lay;        // the rebuild: A, B and the layout's buffers, filled here
    const uint8_t *src;    // old contents: the table itself, or its snapshot
    const uint8_t *src2;   // second table of a merge, or null
    uint8_t *snap;         // in-place first: where the snapshot goes (src too), or null
    uint32_t *fused_fail;  // zero; set by the in-place phase
    int lists_only;        // stop before the layout (which is queued behind, with the whole GPU)
    const uint32_t *keys;  // the batch (n = 0 in a merge, or when it is bucketed already)
    uint32_t n, nbytes;
    Counts3 *tiles;
    uint32_t *Q, *E, *E2, *abase, *acnt, *bbase, *b2cnt, *bcnt, *bfill, *bitems;
    uint32_t *dups;  // set when the table holds copies
    uint32_t *bar;   // four zero words
};

// Exclusive scans of NV interleaved words per entry by one CTA of FB_THREADS
// threads, each a contiguous stretch of entries.
template <int NV>
__device__ __forceinline__ void fb_scan(const uint32_t *in, uint32_t *out, uint32_t n, bool total)
{
    __shared__ uint32_t s_w[NV][FB_THREADS / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t per = (n + FB_THREADS - 1) / FB_THREADS;
    const uint32_t i0 = min(n, tid * per), i1 = min(n, i0 + per);
    uint32_t run[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) run[v] = 0;
    for (uint32_t i = i0; i < i1; i++) {
#pragma unroll
        for (int v = 0; v < NV; v++) run[v] += __ldcg(in + NV * i + v);
    }
#pragma unroll
    for (int v = 0; v < NV; v++) {
        uint32_t incl = run[v];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane >= o) incl += x;
        }
        if (lane == 31) s_w[v][wid] = incl;
        run[v] = incl - run[v];
    }
    __syncthreads();
#pragma unroll
    for (int v = 0; v < NV; v++)
        for (uint32_t w = 0; w < wid; w++) run[v] += s_w[v][w];
    for (uint32_t i = i0; i < i1; i++) {
#pragma unroll
        for (int v = 0; v < NV; v++) {
            const uint32_t x = __ldcg(in + NV * i + v);
            out[NV * i + v] = run[v];
            run[v] += x;
        }
    }
    // (the last thread's sums are the totals: a thread without entries keeps its entry sums)
    if (total && tid == FB_THREADS - 1) {
#pragma unroll
        for (int v = 0; v < NV; v++) out[NV * n + v] = run[v];
    }
}

// Leaves of bucket b's batch what changes the table: of deletes as many as
// there are copies, of inserts the first of each new fingerprint.  For buckets
// that a batch with a repeated key or of many times the table's size would take
// past FB_CAP.  (One-byte slots: 18 bits of fingerprint in a bucket.)
__device__ __forceinline__ void fb_reduce(const LayoutArgs &a, uint32_t b, uint32_t *items, uint32_t *cnt)
{
    extern __shared__ __align__(16) uint8_t smem_layout[];
    uint32_t *s_words = reinterpret_cast<uint32_t *>(smem_layout);
    __shared__ uint32_t s_kept;
    constexpr uint32_t FP_BITS = FB_TB + 5, WORDS = 1u << (FP_BITS - 5);
    const uint32_t tid = threadIdx.x, na = a.A.count(b), n = a.B.count(b);
    const uint32_t *A = a.A.items + a.A.start(b);
    uint32_t *B = items + a.B.start(b);
    const bool del = a.op == OP_DELETE;
    if (del && na > 2 * WORDS) return;  // (a counter of 16 bits per stored element)
    for (uint32_t i = tid; i < WORDS; i += FB_THREADS) s_words[i] = 0;
    if (tid == 0) s_kept = 0;
    __syncthreads();
    for (uint32_t i0 = 0; i0 < n; i0 += FB_THREADS) {
        const uint32_t i = i0 + tid, fp = i < n ? __ldcg(B + i) : 0u;
        bool keep = false;
        if (i < n) {
            uint32_t lo = 0, hi = na;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (A[mid] < fp) lo = mid + 1;
                else hi = mid;
            }
            const bool stored = lo < na && A[lo] == fp;
            if (del && stored) {
                const uint32_t sh = 16 * (lo & 1u);
                uint32_t c = (*reinterpret_cast<volatile uint32_t *>(s_words + (lo >> 1)) >> sh) & 0xFFFFu;
                if (lo + c < na && A[lo + c] == fp) {
                    c = (atomicAdd(s_words + (lo >> 1), 1u << sh) >> sh) & 0xFFFFu;
                    keep = lo + c < na && A[lo + c] == fp;
                }
            } else if (!del && !stored) {
                const uint32_t x = fp & ((1u << FP_BITS) - 1u), bit = 1u << (x & 31u);
                keep = !(atomicOr(s_words + (x >> 5), bit) & bit);
            }
        }
        __syncthreads();  // the 256 items are read; places at or before them are written
        if (keep) B[atomicAdd(&s_kept, 1u)] = fp;
        __syncthreads();
    }
    if (tid == 0) cnt[b] = s_kept;
    __syncthreads();
}

template <int BPE>
__global__ void __launch_bounds__(FB_THREADS, 2) k_update_fallback(FallbackArgs f)
{
    if (!(*f.gate & f.gate_bits)) return;
    extern __shared__ __align__(16) uint8_t smem_layout[];
    uint32_t *s_out = reinterpret_cast<uint32_t *>(smem_layout);
    __shared__ uint32_t s_u;
    const LayoutArgs &a = f.lay;
    const uint32_t tid = threadIdx.x, gt = blockIdx.x * FB_THREADS + tid, gn = gridDim.x * FB_THREADS;
    const uint32_t ntiles = (a.nslots + EXTRACT_TILE - 1) / EXTRACT_TILE;
    const uint32_t shift = a.r + a.tb, mask = (1u << (a.q + a.r)) - 1u;
    // what the layouts expect at zero
    auto reset = [&]() {
        for (uint32_t b = gt; b < a.nb; b += gn) a.status[b] = 0ull;
        if (gt == 0) *a.ticket = *a.fix_cnt = *f.dups = 0u;
    };
    auto buckets = [&](auto &&body) {
        for (;;) {
            __syncthreads();
            if (tid == 0) s_u = atomicAdd(a.ticket, 1u);
            __syncthreads();
            const uint32_t b = s_u;
            if (b >= a.nb) break;
            body(b);
        }
    };
    reset();
    if (f.n)
        for (uint32_t b = gt; b < a.nb; b += gn) f.bcnt[b] = f.bfill[b] = 0u;
    if (f.snap) {
        const uint4 *t = reinterpret_cast<const uint4 *>(a.table);
        for (uint32_t i = gt; i < f.nbytes / 16; i += gn) reinterpret_cast<uint4 *>(f.snap)[i] = t[i];
        for (uint32_t i = (f.nbytes & ~15u) + gt; i < f.nbytes; i += gn) f.snap[i] = a.table[i];
    }
    if (!grid_sync(f.bar, a.err)) return;
    if (gt == 0) *a.err = 0u;  // (it may be the gate: every CTA has looked at it)
    // the batch's fingerprints by bucket
    if (f.n) {
        for (uint32_t i = gt; i < f.n; i += gn) atomicAdd(f.bcnt + ((aphash32(f.keys[i]) & mask) >> shift), 1u);
        if (!grid_sync(f.bar, a.err)) return;
        if (blockIdx.x == 0) fb_scan<1>(f.bcnt, f.bbase, a.nb, false);
        if (!grid_sync(f.bar, a.err)) return;
        for (uint32_t i = gt; i < f.n; i += gn) {
            const uint32_t fp = aphash32(f.keys[i]) & mask, b = fp >> shift;
            f.bitems[f.bbase[b] + atomicAdd(f.bfill + b, 1u)] = fp;
        }
    }
    if constexpr (BPE == 1) {
        if (f.snap) {
            LayoutArgs u = a;
            u.A = BucketSrc{nullptr, nullptr, 0, nullptr};
            u.B = BucketSrc{f.bitems, f.bbase, 0, f.bcnt};
            u.src_table = f.snap;
            u.fused_fail = f.fused_fail;
            for (uint32_t i = (1u << a.q) + gt; i < f.nbytes; i += gn) a.table[i] = 0;
            if (!grid_sync(f.bar, a.err)) return;
            if (a.op == OP_DELETE) buckets([&](uint32_t b) { bucket_layout_set<FB_THREADS, 32, OwnLessTable>(u, b); });
            else buckets([&](uint32_t b) { bucket_layout_set<FB_THREADS, 32, OwnTable>(u, b); });
            if (!grid_sync(f.bar, a.err)) return;
            if (!__ldcg(f.fused_fail)) {
                const uint32_t nf = min(__ldcg(a.fix_cnt), a.fix_cap);
                for (uint32_t i = gt; i < nf; i += gn) a.table[__ldcg(a.fix_list + i)] |= 4u;
                return;
            }
            if (!grid_sync(f.bar, a.err)) return;  // (all have read the flag and the count)
            reset();
            if (gt == 0) *a.err = 0u;
        }
    }
    // the old contents as sorted lists, with the buckets' bounds
    for (int k = 0; k < (f.src2 ? 2 : 1); k++) {
        const uint8_t *src = k ? f.src2 : f.src;
        uint32_t *E = k ? f.E2 : f.E, *base = k ? f.bbase : f.abase, *cnt = k ? f.b2cnt : f.acnt;
        if (!grid_sync(f.bar, a.err)) return;
        for_each_tile(a.nslots, [&](uint32_t u) { tile_counts<BPE, false>(u, src, a.nslots, f.nbytes, f.tiles, k ? nullptr : f.dups); });
        if (!grid_sync(f.bar, a.err)) return;
        if (blockIdx.x == 0)
            fb_scan<3>(reinterpret_cast<const uint32_t *>(f.tiles), reinterpret_cast<uint32_t *>(f.tiles), ntiles, true);
        if (!grid_sync(f.bar, a.err)) return;
        for_each_tile(a.nslots, [&](uint32_t u) { occ_list<BPE, false>(u, src, a.nslots, f.nbytes, f.tiles, f.Q, s_out); });
        if (!grid_sync(f.bar, a.err)) return;
        for_each_tile(a.nslots, [&](uint32_t u) { extract<BPE, false>(u, src, a.nslots, f.nbytes, a.r, f.tiles, f.Q, E, s_out); });
        if (!grid_sync(f.bar, a.err)) return;
        const uint32_t m = f.tiles[ntiles].ne;
        auto lower = [&](uint32_t b) -> uint32_t {
            const uint64_t key = (uint64_t)b << shift;
            uint32_t lo = 0, hi = m;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if ((uint64_t)E[mid] < key) lo = mid + 1;
                else hi = mid;
            }
            return lo;
        };
        for (uint32_t b = gt; b < a.nb; b += gn) {
            const uint32_t lo = lower(b);
            base[b] = lo;
            cnt[b] = lower(b + 1) - lo;
        }
    }
    // the slots past the last bucket's quotients only receive spill
    for (size_t i = ((size_t)BPE << a.q) + gt; i < f.nbytes; i += gn) a.table[i] = 0;
    if (f.lists_only) return;
    if (!grid_sync(f.bar, a.err)) return;
    // (the set layout's map of a bucket reaches its last quotient: whole
    // buckets only)
    if (BPE == 1 && a.q >= a.tb && (a.op == OP_MERGE || !__ldcg(f.dups))) {
        if (a.op == OP_DELETE) buckets([&](uint32_t b) { bucket_layout_set<FB_THREADS, 32, OwnLessSource>(a, b); });
        else buckets([&](uint32_t b) { bucket_layout_set<FB_THREADS, 32, OwnListSource>(a, b); });
    } else {
        buckets([&](uint32_t b) {
            if (BPE == 1 && f.n && a.A.count(b) + a.B.count(b) > FB_CAP) fb_reduce(a, b, f.bitems, f.bcnt);
            bucket_layout_body<FB_THREADS, 32, BPE>(a, b);
        });
    }
    if (!grid_sync(f.bar, a.err)) return;
    const uint32_t nf = min(__ldcg(a.fix_cnt), a.fix_cap);
    for (uint32_t i = gt; i < nf; i += gn) a.table[(size_t)__ldcg(a.fix_list + i) * BPE + (BPE - 1)] |= 4u;
}

}  // namespace gqf

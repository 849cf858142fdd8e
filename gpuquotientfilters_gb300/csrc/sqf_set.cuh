// Item-parallel bucket layouts.  One-byte slots with no fingerprint stored
// twice (r = 5): builds and merges from fingerprint lists (k_set_layout),
// and the in-place merge and large insert, which decode a bucket's old
// contents straight from the table (k_set_update).  Builds and merges that
// keep every copy, or of two-byte slots: k_group_layout.
#pragma once

#include "sqf_build.cuh"

namespace gqf {

// ---------------------------------------------------------------------
// Set layout (one-byte slots, r = 5, set semantics).  The bucket's
// fingerprints are one u32 remainder set per quotient; every quotient's run
// start is computed once and kept as a one-byte displacement from its home
// slot, and then every ITEM writes its own slot: run start + number of
// smaller remainders in its quotient's set.  The items come a second time
// from their list (still in L2), 16 bytes a load, so all lanes of a warp do
// the same work whatever the quotients hold.  Repeated fingerprints write the
// same byte twice.
//
// The displacements are first computed as if nothing spilled in from the
// bucket before, and warp 0 looks back for the true entry slot while the
// other warps write the items.  A spill changes only the leading quotients
// up to the first gap it fits in; those are then laid out again, one warp
// per 32 of them.
// ---------------------------------------------------------------------
constexpr uint32_t SET_R = 5;
constexpr uint32_t SET_SPILL = 2048;   // tile slots past the bucket; the rest goes straight to the table
constexpr uint32_t SET_ESCAPE = 255;   // displacement that does not fit a byte: recomputed from the thread's start

// Shared memory of a layout CTA: run displacements, tile, occupied bits, the
// threads' first free slots, then the bucket's contents.
struct ItemsPlan {
    size_t tile, occ, gc, contents;
};
__host__ __device__ constexpr ItemsPlan items_plan(size_t S, size_t threads, size_t bpe)
{
    ItemsPlan m{};
    m.tile = (S + 15) & ~(size_t)15;
    m.occ = m.tile + (S + SET_SPILL) * bpe + 16;
    m.gc = m.occ + ((S / 8 + 15) & ~(size_t)15);
    m.contents = m.gc + 4 * (threads + 4);
    return m;
}
__host__ __device__ inline size_t set_layout_smem(uint32_t tb, uint32_t threads)  // remainder sets
{
    return items_plan((size_t)1 << tb, threads, 1).contents + ((size_t)4 << tb);
}

// Shared-memory byte offset of the remainder set of local quotient x: the
// eight 16-byte words of 32 quotients are permuted by the index of the 32,
// so threads reading their own 32 quotients, 128 bytes apart, hit distinct
// banks.
__device__ __forceinline__ uint32_t set_addr(uint32_t x) { return (x << 2) ^ ((x >> 1) & 0x70u); }

// f(item) for n items from items[start] (items 16-byte aligned), shared by
// NT threads of which this is number t: single items up to the first and
// from the last 16-byte boundary, 16-byte loads between.
template <int NT, bool NC = true, typename F>
__device__ __forceinline__ void for_each_item(const uint32_t *items, size_t start, uint32_t n,
                                              uint32_t t, F &&f)
{
    const uint32_t head = min(n, (uint32_t)(-(uint32_t)start & 3u)), nv = (n - head) >> 2, tail = head + 4 * nv;
    const uint32_t *it = items + start;
    const uint4 *v4 = reinterpret_cast<const uint4 *>(it + head);
    for (uint32_t j = t; j < nv; j += 2 * NT) {  // two loads in flight per thread
        const bool two = j + NT < nv;
        const uint4 a = ld_data<NC>(v4 + j), b = two ? ld_data<NC>(v4 + j + NT) : make_uint4(0, 0, 0, 0);
        f(a.x);
        f(a.y);
        f(a.z);
        f(a.w);
        if (two) {
            f(b.x);
            f(b.y);
            f(b.z);
            f(b.w);
        }
    }
    if (t < head) f(ld_data<NC>(it + t));
    if (t < n - tail) f(ld_data<NC>(it + tail + t));
}

// One step of the layout map over consecutive quotients, relative to the
// current quotient: u = first free slot - quotient.  A quotient with k items
// starts its run max(u, 0) slots past home; the next one sees
// u' = max(u, 0) + k - 1.  (A quotient without items leaves the first free
// slot at its own home if it was below; no later quotient can tell.)
__device__ __forceinline__ int set_step(int u, int k) { return __viaddmax_s32(u, k - 1, k - 1); }

// The bucket's fingerprints from lists: A (a table's extracted contents) and
// B (the batch).  DELETES: the batch is taken out.  NC: the lists are older
// than the launch.
template <int THREADS, int QPT, bool DELETES, bool NC>
struct Lists {
    static constexpr bool DEL = DELETES;
    static constexpr uint32_t S = THREADS * QPT;
    const LayoutArgs &a;
    uint32_t na, nb;
    size_t abase, bbase;
    __device__ __forceinline__ Lists(const LayoutArgs &args, uint32_t b, uint8_t *) : a(args)
    {
        na = a.A.count(b);
        nb = a.B.count(b);
        abase = na ? a.A.start(b) : 0;
        bbase = nb ? a.B.start(b) : 0;
    }
    __device__ __forceinline__ void index() {}
    // every fingerprint of the table, then those of the batch (local
    // quotient, remainder), shared by NT threads of which this is number t
    template <int NT, typename F>
    __device__ __forceinline__ void table_items(uint32_t t, F &&f) const
    {
        if (na) for_each_item<NT, NC>(a.A.items, abase, na, t, [&](uint32_t v) { f((v >> SET_R) & (S - 1), v & 31u); });
    }
    template <int NT, typename F>
    __device__ __forceinline__ void batch_items(uint32_t t, F &&f) const
    {
        for_each_item<NT, NC>(a.B.items, bbase, nb, t, [&](uint32_t v) { f((v >> SET_R) & (S - 1), v & 31u); });
    }
};
template <int THREADS, int QPT>
using ListSource = Lists<THREADS, QPT, false, true>;
template <int THREADS, int QPT>
using OwnListSource = Lists<THREADS, QPT, false, false>;
template <int THREADS, int QPT>
using OwnLessSource = Lists<THREADS, QPT, true, false>;

// Contents of a bucket as remainder sets, fed by a source (lists, or tables).
template <int THREADS, int QPT, template <int, int> class Source>
struct SetContents {
    static constexpr int BPE = 1;
    static constexpr bool SMALL = true;  // at most 32 items a quotient
    static constexpr bool DEL = Source<THREADS, QPT>::DEL;
    static constexpr uint32_t S = THREADS * QPT;
    uint8_t *mask;  // u32 at set_addr(x)
    Source<THREADS, QPT> src;
    __device__ __forceinline__ SetContents(const LayoutArgs &a, uint32_t b, uint8_t *mem) : mask(mem), src(a, b, mem + 4 * S) {}
    __device__ __forceinline__ uint32_t &at(uint32_t x) const { return *reinterpret_cast<uint32_t *>(mask + set_addr(x)); }
    __device__ __forceinline__ bool fits() const { return true; }
    __device__ __forceinline__ void load()
    {
        for (uint32_t i = threadIdx.x; i < S / 4; i += THREADS) reinterpret_cast<uint4 *>(mask)[i] = make_uint4(0, 0, 0, 0);
        src.index();
        __syncthreads();
        if constexpr (DEL) {  // a table without copies loses the batch's fingerprints
            src.template table_items<THREADS>(threadIdx.x, [&](uint32_t x, uint32_t rem) { atomicOr(&at(x), 1u << rem); });
            __syncthreads();
            src.template batch_items<THREADS>(threadIdx.x, [&](uint32_t x, uint32_t rem) { atomicAnd(&at(x), ~(1u << rem)); });
        } else {
            each<THREADS>(threadIdx.x, [&](uint32_t x, uint32_t rem) { atomicOr(&at(x), 1u << rem); });
        }
        __syncthreads();
    }
    __device__ __forceinline__ void sizes(uint32_t x, uint32_t (&k)[4]) const  // of quotients x .. x + 3
    {
        const uint4 m = *reinterpret_cast<const uint4 *>(mask + set_addr(x));
        k[0] = __popc(m.x);
        k[1] = __popc(m.y);
        k[2] = __popc(m.z);
        k[3] = __popc(m.w);
    }
    __device__ __forceinline__ uint32_t size(uint32_t x) const { return __popc(at(x)); }
    template <int NT, typename F>
    __device__ __forceinline__ void each(uint32_t t, F &&f) const
    {
        src.template table_items<NT>(t, f);
        if (!DEL) src.template batch_items<NT>(t, f);
    }
    // put(slot, element) for an item of a run that starts at slot st; the
    // element's occupied bit is not set
    template <typename Put>
    __device__ __forceinline__ void put_item(uint32_t x, uint32_t rem, uint32_t st, Put &&put) const
    {
        const uint32_t m = at(x), below = __popc(m & ((1u << rem) - 1u)), p = st + below;
        if (DEL && !((m >> rem) & 1u)) return;
        put(p, (rem << 3) + 2 * min(below, 1u) + min(p - x, 1u));
    }
    template <typename Put>
    __device__ __forceinline__ void put_run(uint32_t x, uint32_t st, Put &&put) const
    {
        uint32_t f = 0;
        for (uint32_t m = at(x); m; m &= m - 1u, st++, f = 2u) put(st, ((__ffs(m) - 1) << 3) + f + min(st - x, 1u));
    }
    template <int NT, typename Start, typename Put>
    __device__ __forceinline__ void put_big(uint32_t, Start &&, Put &&) const
    {
    }
};

// Contents of a bucket as groups: the remainders of each quotient next to
// each other (counting sort), in any order.  Every copy is kept, or (UNIQUE)
// repeats are struck out.  An item's slot is its run's start plus the smaller
// ones of its group; equal copies each write all of their slots.  Groups of
// more than BIG items are sorted and laid out by one thread each instead.  A
// bucket with more items than the shared memory was sized for keeps its
// remainders in global scratch.
//
// A thread sorting and walking its 32 quotients' groups one after the other
// took 396 us for 12.3M fingerprints over 2^24 quotients; this took 172 us.
// Loops over a group (one to three items) are not unrolled: that build as a
// whole took 276 us unrolled and takes 249, and compiles in a third of the time.
template <int THREADS, int QPT, int BPE_, bool UNIQUE>
struct GroupContents {
    static constexpr int BPE = BPE_;
    static constexpr bool SMALL = false;
    static constexpr uint32_t S = THREADS * QPT, R = BPE == 1 ? 5 : 13, BIG = 48;
    using Rem = typename std::conditional<BPE == 1, uint8_t, uint16_t>::type;
    static constexpr uint32_t STRUCK = BPE == 1 ? 0xFFu : 0xFFFFu;  // above every remainder
    const LayoutArgs &a;
    uint32_t *cnt;  // u16 per quotient: end of its group
    Rem *rem;
    uint32_t n, na;
    size_t abase, bbase;
    __device__ __forceinline__ GroupContents(const LayoutArgs &args, uint32_t b, uint8_t *mem) : a(args)
    {
        na = a.A.count(b);
        n = na + a.B.count(b);
        abase = na ? a.A.start(b) : 0;
        bbase = n > na ? a.B.start(b) : 0;
        cnt = reinterpret_cast<uint32_t *>(mem);
        // (the lists before this bucket's hold A.start + B.start items)
        rem = n <= a.cap_items ? reinterpret_cast<Rem *>(mem + group_cnt_bytes(S))
                               : static_cast<Rem *>(a.rem_scratch) +
                                     ((a.A.cnt ? a.A.start(b) : 0) + (a.B.cnt ? a.B.start(b) : 0));
    }
    static __host__ __device__ constexpr size_t group_cnt_bytes(size_t s) { return (4 * (s / 2 + s / 32 + 8) + 15) & ~(size_t)15; }
    __device__ __forceinline__ bool fits() const { return n <= 65520; }  // u16 positions
    __device__ __forceinline__ uint32_t end(uint32_t x) const { return cnt16_get(cnt, x); }
    __device__ __forceinline__ uint32_t begin(uint32_t x) const { return x ? cnt16_get(cnt, x - 1) : 0u; }
    __device__ __forceinline__ void load()
    {
        __shared__ uint32_t s_w[THREADS / 32];
        const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
#pragma unroll 1
        for (uint32_t i = tid; i < S / 2 + S / 32 + 8; i += THREADS) cnt[i] = 0;
        __syncthreads();
        each<THREADS>(tid, [&](uint32_t x, uint32_t) { cnt16_fetch_inc(cnt, x); });
        __syncthreads();
        uint32_t sum = 0;
        for (uint32_t j = 0; j < QPT; j += 2) {
            const uint32_t c = cnt[skew16((tid * QPT + j) >> 1)];
            sum += (c & 0xFFFFu) + (c >> 16);
        }
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane >= o) incl += v;
        }
        if (lane == 31) s_w[wid] = incl;
        __syncthreads();
        uint32_t run = incl - sum;
        for (uint32_t w = 0; w < wid; w++) run += s_w[w];
        for (uint32_t j = 0; j < QPT; j += 2) {  // both counters of a word
            const uint32_t w = skew16((tid * QPT + j) >> 1), c = cnt[w], c0 = c & 0xFFFFu;
            cnt[w] = run | ((run + c0) << 16);
            run += c0 + (c >> 16);
        }
        __syncthreads();
        each<THREADS>(tid, [&](uint32_t x, uint32_t r) { rem[cnt16_fetch_inc(cnt, x)] = (Rem)r; });
        __syncthreads();
#pragma unroll 1
        for (uint32_t x = tid; x < S; x += THREADS) {
            const uint32_t g0 = begin(x), g1 = end(x);
            if (g1 - g0 < 2) continue;
            if (g1 - g0 > BIG) {
                small_sort(rem + g0, g1 - g0);
                if (UNIQUE) {
                    uint32_t k = g0 + 1;
#pragma unroll 1
                    for (uint32_t i = g0 + 1; i < g1; i++)
                        if (rem[i] != rem[k - 1]) rem[k++] = rem[i];
                    for (; k < g1; k++) rem[k] = (Rem)STRUCK;
                }
            } else if (UNIQUE) {
#pragma unroll 1
                for (uint32_t i = g0 + 1; i < g1; i++) {
                    const Rem v = rem[i];
#pragma unroll 1
                    for (uint32_t j = g0; j < i; j++)
                        if (rem[j] == v) {
                            rem[i] = (Rem)STRUCK;
                            break;
                        }
                }
            }
        }
        __syncthreads();
    }
    __device__ __forceinline__ uint32_t kept(uint32_t g0, uint32_t g1) const
    {
        if (!UNIQUE || g1 - g0 < 2) return g1 - g0;
        uint32_t k = 0;
#pragma unroll 1
        for (uint32_t i = g0; i < g1; i++) k += rem[i] != (Rem)STRUCK ? 1u : 0u;
        return k;
    }
    __device__ __forceinline__ void sizes(uint32_t x, uint32_t (&k)[4]) const
    {
        uint32_t g = begin(x);
        const uint32_t w0 = cnt[skew16(x >> 1)], w1 = cnt[skew16((x >> 1) + 1)];
        const uint32_t e[4] = {w0 & 0xFFFFu, w0 >> 16, w1 & 0xFFFFu, w1 >> 16};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            k[i] = kept(g, e[i]);
            g = e[i];
        }
    }
    __device__ __forceinline__ uint32_t size(uint32_t x) const { return kept(begin(x), end(x)); }
    template <int NT, typename F>
    __device__ __forceinline__ void each(uint32_t t, F &&f) const
    {
        auto item = [&](uint32_t v) { f((v >> R) & (S - 1), v & ((1u << R) - 1u)); };
        if (na) for_each_item<NT>(a.A.items, abase, na, t, item);
        if (n > na) for_each_item<NT>(a.B.items, bbase, n - na, t, item);
    }
    template <typename Put>
    __device__ __forceinline__ void put_item(uint32_t x, uint32_t r, uint32_t st, Put &&put) const
    {
        const uint32_t g0 = begin(x), g1 = end(x);
        uint32_t less = 0, same = 1;
        if (g1 - g0 > 1) {
            if (g1 - g0 > BIG) return;  // put_big
            same = 0;
#pragma unroll 1
            for (uint32_t i = g0; i < g1; i++) {
                less += rem[i] < (Rem)r ? 1u : 0u;
                same += rem[i] == (Rem)r ? 1u : 0u;
            }
        }
#pragma unroll 1
        for (uint32_t k = less; k < less + same; k++)
            put(st + k, (r << 3) + 2 * min(k, 1u) + min(st + k - x, 1u));
    }
    template <typename Put>
    __device__ __forceinline__ void put_run(uint32_t x, uint32_t st, Put &&put) const
    {
        const uint32_t g0 = begin(x), g1 = end(x);
        const bool sorted = g1 - g0 > BIG;
#pragma unroll 1
        for (uint32_t i = g0; i < g1; i++) {
            const uint32_t r = rem[i];
            if (UNIQUE && r == STRUCK) continue;
            uint32_t k = i - g0;
            if (!sorted) {
                k = 0;
#pragma unroll 1
                for (uint32_t j = g0; j < g1; j++) k += (rem[j] < (Rem)r || (rem[j] == (Rem)r && j < i)) ? 1u : 0u;
            }
            put(st + k, (r << 3) + 2 * min(k, 1u) + min(st + k - x, 1u));
        }
    }
    // the groups put_item leaves out
    template <int NT, typename Start, typename Put>
    __device__ __forceinline__ void put_big(uint32_t t, Start &&start, Put &&put) const
    {
#pragma unroll 1
        for (uint32_t x = t; x < S; x += NT)
            if (end(x) - begin(x) > BIG) put_run(x, start(x), put);
    }
};

template <int THREADS, int QPT, class Contents>
__device__ __forceinline__ void bucket_layout_items(const LayoutArgs &a, const uint32_t b)
{
    extern __shared__ __align__(16) uint8_t smem_layout[];
    constexpr int BPE = Contents::BPE;
    // (groups keep nothing in registers between the passes over a thread's
    // quotients; unrolled, each of those kernels took 12 to 20 s to compile)
    constexpr int JUNROLL = Contents::SMALL ? QPT / 4 : 1;
    constexpr uint32_t S = THREADS * QPT, BUF = S + SET_SPILL, NW = THREADS / 32;
    constexpr ItemsPlan pl = items_plan(S, THREADS, BPE);
    uint8_t *s_disp = smem_layout;            // displacement of quotient x's run
    uint8_t *s_tile = smem_layout + pl.tile;  // slot x0 + i at byte BPE * i
    uint32_t *s_occ = reinterpret_cast<uint32_t *>(smem_layout + pl.occ);
    uint32_t *s_gc = reinterpret_cast<uint32_t *>(smem_layout + pl.gc);  // first free slot (from x0) at each thread's quotients
    __shared__ uint32_t s_cin, s_cout, s_nfix, s_fbase, s_naff;
    __shared__ LayoutFn s_wfn[NW];
    __shared__ uint32_t s_fix[256];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t x0 = b * S, qb = tid * QPT;
    Contents con(a, b, smem_layout + pl.contents);
    if (!con.fits()) {  // flag it and keep the chain alive
        if (tid == 0) {
            atomicOr(a.err, DEV_ERR_BUCKET_CAP);
            st_relaxed_u64(a.status + b, lb_pack_inc(x0));
        }
        return;
    }
    auto fix_lost = [&]() {
        if (a.fused_fail) atomicOr(a.fused_fail, 1u);
        else if (!a.fix_soft) atomicOr(a.err, DEV_ERR_BUCKET_CAP);
    };
    auto put_tile = [&](uint32_t p, uint32_t e) {
        if (p >= BUF) return;
        if (BPE == 1) s_tile[p] = (uint8_t)e;
        else reinterpret_cast<uint16_t *>(s_tile)[p] = (uint16_t)__byte_perm(e, 0, 0x4401);
    };

    if (tid == 0) {
        s_nfix = 0;
        s_naff = 0;
    }
    for (uint32_t i = tid; i < BUF * BPE / 16; i += THREADS)
        reinterpret_cast<uint4 *>(s_tile)[i] = make_uint4(0, 0, 0, 0);
    if (QPT < 32)
        for (uint32_t i = tid; i < (S + 31) / 32; i += THREADS) s_occ[i] = 0;
    con.load();

    // this thread's quotients: sizes (one per byte), occupied bits, map
    uint32_t kk[QPT / 4], nz = 0;
    LayoutFn fn{0u, 0u};
    {
        int u = -1;  // entering below the first quotient
#pragma unroll(JUNROLL)
        for (uint32_t j4 = 0; j4 < QPT / 4; j4++) {
            uint32_t k[4];
            con.sizes(qb + 4 * j4, k);
#pragma unroll
            for (int e = 0; e < 4; e++) u = set_step(u, (int)k[e]);
            if constexpr (Contents::SMALL) {
                const uint32_t pk = k[0] + (k[1] << 8) + (k[2] << 16) + (k[3] << 24);
                kk[j4] = pk;
                fn.n = __dp4a(pk, 0x01010101u, fn.n);
                const uint32_t f = ((pk + 0x7F7F7F7Fu) >> 7) & 0x01010101u;  // byte e: quotient e has items
                nz |= ((f * 0x01020408u) >> 24 & 15u) << (4 * j4);
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    fn.n += k[e];
                    nz |= (k[e] ? 1u : 0u) << (4 * j4 + e);
                }
            }
        }
        fn.F = (uint32_t)((int)(x0 + qb + QPT) + u);
    }
    // maps of the threads before this one, in the warp and then the CTA
    LayoutFn pre, all;
    {
        LayoutFn f = fn;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            LayoutFn pv;
            pv.n = __shfl_up_sync(0xffffffffu, f.n, o);
            pv.F = __shfl_up_sync(0xffffffffu, f.F, o);
            if (lane >= o) f = compose(pv, f);
        }
        pre.n = __shfl_up_sync(0xffffffffu, f.n, 1);
        pre.F = __shfl_up_sync(0xffffffffu, f.F, 1);
        if (lane == 0) pre = LayoutFn{0u, 0u};
        if (lane == 31) s_wfn[wid] = f;
    }
    __syncthreads();
    {
        LayoutFn f{0u, 0u};
        if (lane < (int)NW) f = s_wfn[lane];
#pragma unroll
        for (int o = 1; o < (int)NW; o <<= 1) {
            LayoutFn pv;
            pv.n = __shfl_up_sync(0xffffffffu, f.n, o);
            pv.F = __shfl_up_sync(0xffffffffu, f.F, o);
            if (lane >= o) f = compose(pv, f);
        }
        all.n = __shfl_sync(0xffffffffu, f.n, NW - 1);
        all.F = __shfl_sync(0xffffffffu, f.F, NW - 1);
        LayoutFn wpre;
        wpre.n = __shfl_sync(0xffffffffu, f.n, wid ? wid - 1 : 0);
        wpre.F = __shfl_sync(0xffffffffu, f.F, wid ? wid - 1 : 0);
        if (wid) pre = compose(wpre, pre);
    }
    if (tid == 0) {
        if (all.n > LB_VMAX / 2 || all.F > LB_VMAX / 2) atomicOr(a.err, DEV_ERR_FULL);
        if (b != 0) st_relaxed_u64(a.status + b, lb_pack_agg(all.n, all.F));
    }
    // displacements from a first free slot c at this thread's quotients
    auto displace = [&](uint32_t c) {
        s_gc[tid] = c - x0;
        int u = (int)c - (int)(x0 + qb);
#pragma unroll(JUNROLL)
        for (uint32_t j4 = 0; j4 < QPT / 4; j4++) {
            uint32_t pk = 0, k[4];
            if constexpr (Contents::SMALL) {
#pragma unroll
                for (int e = 0; e < 4; e++) k[e] = (kk[j4] >> (8 * e)) & 0xFFu;
            } else {
                con.sizes(qb + 4 * j4, k);
            }
#pragma unroll
            for (uint32_t e = 0; e < 4; e++) {
                const int d = max(u, 0);
                u = d + (int)k[e] - 1;
                pk |= (uint32_t)min(d, (int)SET_ESCAPE) << (8 * e);
            }
            reinterpret_cast<uint32_t *>(s_disp)[(qb >> 2) + j4] = pk;
        }
    };
    const uint32_t cspec = max(pre.apply(x0), x0);  // as if the bucket were entered at x0
    displace(cspec);
    __syncthreads();

    // first slot (from x0) of quotient x's run
    auto start_of = [&](uint32_t x) -> uint32_t {
        const uint32_t d = s_disp[x];
        if (d != SET_ESCAPE) return x + d;
        const uint32_t y0 = x & ~(uint32_t)(QPT - 1);  // walk the thread's quotients up to x
        int u = (int)s_gc[x / QPT] - (int)y0;
        for (uint32_t y = y0; y < x; y++) u = set_step(u, (int)con.size(y));
        return x + (uint32_t)max(u, 0);
    };
    if (wid == 0) {
        uint32_t cin = 0;
        if (b != 0) cin = lookback_cin_warp(a.status, b, a.err);
        const uint32_t cout = all.apply(cin);
        if (lane == 0) {
            st_relaxed_u64(a.status + b, lb_pack_inc(cout));
            s_cin = cin;
            s_cout = cout;
        }
    }
    if (NW == 1 || wid > 0) {
        // every item writes its slot of the tile
        constexpr int NT = NW == 1 ? THREADS : THREADS - 32;
        const uint32_t t = NW == 1 ? tid : tid - 32;
        con.template each<NT>(t, [&](uint32_t x, uint32_t rem) { con.put_item(x, rem, start_of(x), put_tile); });
        con.template put_big<NT>(t, start_of, put_tile);
    }
    __syncthreads();
    const uint32_t cin = s_cin, cout = s_cout;
    const uint32_t lo = cin > x0 ? cin : x0;
    uint32_t hi = cout > x0 + S ? cout : x0 + S;
    if (hi > a.nslots) {
        if (cout > a.nslots && tid == 0) atomicOr(a.err, DEV_ERR_FULL);
        hi = a.nslots;
    }
    const uint32_t lo_l = lo - x0, hi_l = hi > x0 ? hi - x0 : 0u;
    const uint32_t lim = hi_l < BUF ? hi_l : BUF;  // slots the tile holds
    if (lo_l) {
        // entered past x0: the threads whose first free slot moves (a
        // leading range of threads) lay their quotients out again
        const uint32_t c = max(pre.apply(cin), lo);
        const bool aff = c != cspec;
        const unsigned am = __ballot_sync(0xffffffffu, aff);
        if (am && lane == 0) atomicMax(&s_naff, 32u * wid + 32u - (uint32_t)__clz(am));
        if (aff) displace(c);
        __syncthreads();
        const uint32_t naff = s_naff;
        // their slots end where the first unmoved thread's begin
        const uint32_t zend = naff < THREADS ? min(s_gc[naff], BUF) : BUF;
        for (uint32_t i = tid; i < zend * BPE; i += THREADS) s_tile[i] = 0;
        __syncthreads();
        for (uint32_t y0 = 32 * wid; y0 < naff * QPT; y0 += THREADS) {
            const uint32_t x = y0 + lane;
            if (x < naff * QPT) con.put_run(x, start_of(x), put_tile);
        }
    }
    // occupied bits; those below lo (their slot was written by an earlier
    // bucket) as fix-ups
    {
        const uint32_t xb = x0 + qb;
        const uint32_t nbelow = lo > xb ? min(lo - xb, (uint32_t)QPT) : 0u;
        const uint32_t bmask = nbelow >= 32u ? 0xFFFFFFFFu : ((1u << nbelow) - 1u);
        for (uint32_t fx = nz & bmask; fx; fx &= fx - 1u) {
            const uint32_t xa = xb + (uint32_t)__ffs(fx) - 1u, p = atomicAdd(&s_nfix, 1u);
            if (p < 256) {
                s_fix[p] = xa;
            } else {
                const uint32_t gp = atomicAdd(a.fix_cnt, 1u);
                if (gp < a.fix_cap) a.fix_list[gp] = xa;
                else fix_lost();
            }
        }
        const uint32_t occ = nz & ~bmask;
        if (QPT >= 32) s_occ[qb >> 5] = occ;
        else if (occ) atomicOr(s_occ + (qb >> 5), occ << (qb & 31));
    }
    if (cout > x0 + BUF) {  // spill past the tile: those items straight to the table
        __syncthreads();
        auto put_far = [&](uint32_t p, uint32_t e) {  // past the table: reported as FULL
            if (p < BUF || p >= hi_l) return;
            uint8_t *d = a.table + ((size_t)x0 + p) * BPE;
            if (BPE == 1) {
                d[0] = (uint8_t)e;
            } else {
                d[0] = (uint8_t)(e >> 8);
                d[1] = (uint8_t)e;
            }
        };
        con.template each<THREADS>(tid, [&](uint32_t x, uint32_t rem) { con.put_item(x, rem, start_of(x), put_far); });
        con.template put_big<THREADS>(tid, start_of, put_far);
    }
    __syncthreads();
    {
        const uint32_t nf = s_nfix < 256 ? s_nfix : 256;
        if (nf) {  // uniform
            if (tid == 0) s_fbase = atomicAdd(a.fix_cnt, nf);
            __syncthreads();
            for (uint32_t i = tid; i < nf; i += THREADS) {
                const uint32_t gp = s_fbase + i;
                if (gp < a.fix_cap) a.fix_list[gp] = s_fix[i];
                else fix_lost();
            }
        }
    }
    // store slots [lo, x0 + lim) with the occupied bits merged in (bit 2 of a
    // slot's last byte): 16-byte words, bytes at a ragged start or end
    constexpr uint32_t SPW = 16 / BPE;  // slots per word
    for (uint32_t g = (lo_l & ~(SPW - 1)) + SPW * tid; g < lim; g += SPW * THREADS) {
        uint4 v = *reinterpret_cast<const uint4 *>(s_tile + g * BPE);
        const uint32_t bits = g < S ? s_occ[g >> 5] >> (g & 31u) : 0u;
        if (BPE == 1) {
            auto spread4 = [](uint32_t x4) -> uint32_t { return ((x4 * 0x00204081u) & 0x01010101u) << 2; };
            v.x |= spread4(bits & 15u);
            v.y |= spread4((bits >> 4) & 15u);
            v.z |= spread4((bits >> 8) & 15u);
            v.w |= spread4((bits >> 12) & 15u);
        } else {
            auto spread2 = [](uint32_t x2) -> uint32_t { return ((x2 & 1u) << 10) | ((x2 & 2u) << 25); };
            v.x |= spread2(bits);
            v.y |= spread2(bits >> 2);
            v.z |= spread2(bits >> 4);
            v.w |= spread2(bits >> 6);
        }
        uint8_t *dst = a.table + ((size_t)x0 + g) * BPE;
        if (g >= lo_l && g + SPW <= lim) {
            *reinterpret_cast<uint4 *>(dst) = v;
        } else {
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            for (uint32_t k = 0; k < 16; k++)
                if (g + k / BPE >= lo_l && g + k / BPE < lim) dst[k] = (uint8_t)(w[k >> 2] >> (8 * (k & 3)));
        }
    }
}
template <int THREADS, int QPT, template <int, int> class Source>
__device__ __forceinline__ void bucket_layout_set(const LayoutArgs &a, const uint32_t b)
{
    bucket_layout_items<THREADS, QPT, SetContents<THREADS, QPT, Source>>(a, b);
}

// ---------------------------------------------------------------------
// The bucket's fingerprints from the table itself (in-place merge, insert and
// delete), and the batch.  Runs are stored in quotient order, one per
// occupied quotient: of the runs starting at or past x0, the first D0 belong
// to quotients below x0 (the lookup's walk back, done once per bucket), the
// next ones to the bucket's occupied quotients in order.  index() keeps, per
// 32-slot word of the slice, its run starts and the run starts before it,
// and the list of the bucket's occupied quotients; then one lane per slot
// finds its run's number by a popcount and its quotient in the list, with
// coalesced byte reads of the slice (L2, L1) in every pass.
// ---------------------------------------------------------------------
__host__ __device__ inline uint32_t upd_spill(uint32_t tb) { return tb >= 12 ? 2048u : 1024u; }
struct SliceIndexPlan {
    size_t rsp, oc, ocp, list, total;
};
__host__ __device__ inline SliceIndexPlan slice_index_plan(uint32_t tb)
{
    const size_t S = (size_t)1 << tb, L = S + upd_spill(tb);
    auto a16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
    SliceIndexPlan m;
    m.rsp = a16(L / 32 * 4);
    m.oc = m.rsp + a16(L / 32 * 2);
    m.ocp = m.oc + a16((S + 31) / 32 * 4);
    m.list = m.ocp + a16((S + 31) / 32 * 2);
    m.total = m.list + a16(S * 2);
    return m;
}

template <int THREADS, int QPT, bool NC>
struct Slice {
    static constexpr uint32_t S = THREADS * QPT;
    const uint8_t *t;
    uint32_t nslots, x0;
    uint32_t *rs32, *oc32;
    uint16_t *rsp, *ocp, *list;
    uint32_t *ctl;  // D0, first slot, end slot, occupied quotients, one past the last non-empty slot

    __device__ __forceinline__ void place(uint8_t *mem, uint32_t tb, uint32_t *c)
    {
        const SliceIndexPlan pl = slice_index_plan(tb);
        rs32 = reinterpret_cast<uint32_t *>(mem);
        rsp = reinterpret_cast<uint16_t *>(mem + pl.rsp);
        oc32 = reinterpret_cast<uint32_t *>(mem + pl.oc);
        ocp = reinterpret_cast<uint16_t *>(mem + pl.ocp);
        list = reinterpret_cast<uint16_t *>(mem + pl.list);
        ctl = c;
    }
    __device__ __forceinline__ uint32_t byte_at(uint32_t i) const  // slot x0 + i
    {
        return x0 + i < nslots ? (uint32_t)ld_data<NC>(t + x0 + i) : 0u;
    }
    // Builds the index.  Returns (on thread 0) whether the slice cannot be
    // decoded; dups: also when a run holds a remainder twice or out of order.
    // s_w: 2 * THREADS / 32 words.  Contains __syncthreads.
    __device__ __forceinline__ bool index(uint32_t *s_w, bool dups)
    {
        constexpr uint32_t NW = THREADS / 32;
        const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
        const uint32_t L = S + upd_spill(31 - __clz(S)), LW = L / 32;
        if (tid == 0) ctl[4] = 0;
        __syncthreads();
        if (wid == 0) {
            const int D = pending_runs_warp<NC>(t, x0);
            if (lane == 0) ctl[0] = (uint32_t)D;
        }
        const uint32_t per = (LW + THREADS - 1) / THREADS;
        const uint32_t w0 = min(LW, tid * per), w1 = min(LW, w0 + per);
        uint32_t cr = 0, co = 0, last = 0;
        uint64_t twice = 0;
        for (uint32_t w = w0; w < w1; w++) {
            uint64_t v[4];
            const uint32_t s0 = x0 + 32 * w;
            if (s0 + 32 <= nslots) {
                const ulonglong2 p0 = ld_data<NC>(reinterpret_cast<const ulonglong2 *>(t + s0));
                const ulonglong2 p1 = ld_data<NC>(reinterpret_cast<const ulonglong2 *>(t + s0) + 1);
                v[0] = p0.x;
                v[1] = p0.y;
                v[2] = p1.x;
                v[3] = p1.y;
            } else {
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    v[h] = 0;
                    for (uint32_t k = 0; k < 8; k++) v[h] |= (uint64_t)byte_at(32 * w + 8 * h + k) << (8 * k);
                }
            }
            uint32_t rsm = 0, ocm = 0, nem = 0;
            uint64_t before = (dups && s0 > 0 && s0 - 1 < nslots) ? (uint64_t)ld_data<NC>(t + s0 - 1) : 0ull;
#pragma unroll
            for (int h = 0; h < 4; h++) {
                const Flags8 f = flags8(v[h]);
                rsm |= (f.nonempty & ~f.cont & 0xFFu) << (8 * h);
                ocm |= (f.occ & 0xFFu) << (8 * h);
                nem |= (f.nonempty & 0xFFu) << (8 * h);
                // bit 7 of a byte: a continuation whose remainder is not above the slot's before it
                const uint64_t prev = (v[h] << 8) | before;
                constexpr uint64_t R5 = 0x1F1F1F1F1F1F1F1Full;
                twice |= ((((prev >> 3) & R5) | BL_HI) - ((v[h] >> 3) & R5)) & (v[h] << 6) & BL_HI;
                before = v[h] >> 56;
            }
            rs32[w] = rsm;
            if (w < (S + 31) / 32) oc32[w] = ocm;
            if (nem) last = 32 * w + (uint32_t)highest_bit(nem) + 1;
            cr += __popc(rsm);
            if (w < (S + 31) / 32) co += __popc(ocm);
        }
        if (last) atomicMax(ctl + 4, last);
        uint32_t ir = cr, io = co;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, ir, o), y = __shfl_up_sync(0xffffffffu, io, o);
            if ((int)lane >= o) {
                ir += x;
                io += y;
            }
        }
        if (lane == 31) {
            s_w[2 * wid] = ir;
            s_w[2 * wid + 1] = io;
        }
        const bool dup = __syncthreads_or(dups && twice != 0);
        const int D0 = (int)ctl[0];
        uint32_t pr = ir - cr, po = io - co, nrs = 0, nocc = 0;
        for (uint32_t w = 0; w < NW; w++) {
            if (w < wid) {
                pr += s_w[2 * w];
                po += s_w[2 * w + 1];
            }
            nrs += s_w[2 * w];
            nocc += s_w[2 * w + 1];
        }
        const uint32_t lastne = ctl[4];
        const bool bad = D0 < 0 || (uint32_t)D0 + nocc > nrs || ((uint32_t)D0 + nocc == nrs && lastne >= L);
        if (tid == 0) {
            ctl[3] = bad ? 0u : nocc;
            if (bad || (uint32_t)D0 >= nrs) ctl[1] = bad ? 0u : lastne;
            if (bad || (uint32_t)D0 + nocc >= nrs) ctl[2] = bad ? 0u : lastne;
        }
        for (uint32_t w = w0; w < w1; w++) {
            const uint32_t rsm = rs32[w], c = __popc(rsm);
            rsp[w] = (uint16_t)pr;
            if (!bad && (uint32_t)D0 - pr < c) ctl[1] = 32 * w + select_bit(rsm, D0 - (int)pr);
            if (!bad && (uint32_t)D0 + nocc - pr < c) ctl[2] = 32 * w + select_bit(rsm, D0 + (int)(nocc - pr));
            pr += c;
            if (w < (S + 31) / 32) {
                ocp[w] = (uint16_t)po;
                po += __popc(oc32[w]);
            }
        }
        __syncthreads();
        for (uint32_t w = wid; w < (S + 31) / 32; w += NW) {
            const uint32_t ow = oc32[w];
            if ((ow >> lane) & 1u) list[ocp[w] + __popc(ow & ((1u << lane) - 1u))] = (uint16_t)(32 * w + lane);
        }
        return bad || dup;
    }
    // f(local quotient, remainder) for every element of the bucket's runs,
    // one lane per slot
    template <int NT, typename F>
    __device__ __forceinline__ void items(uint32_t t0, F &&f) const
    {
        const uint32_t lane = t0 & 31, D0 = ctl[0], nocc = ctl[3], end = ctl[2];
        const uint32_t le = 0xFFFFFFFFu >> (31 - lane);
#pragma unroll 4
        for (uint32_t w = (ctl[1] >> 5) + (t0 >> 5); 32 * w < end; w += NT / 32) {
            const uint32_t e = byte_at(32 * w + lane);
            const uint32_t j = rsp[w] + __popc(rs32[w] & le) - 1u - D0;  // run number among the bucket's
            if ((e & 7u) && j < nocc) f((uint32_t)list[j], e >> 3);
        }
    }
};

// TWO: also the second table of a merge.  DELETES: the batch is taken out.
// NC: the tables and the batch's list are older than the launch.
template <int THREADS, int QPT, bool TWO, bool DELETES, bool NC>
struct TableSource {
    static constexpr bool DEL = DELETES;
    static constexpr uint32_t S = THREADS * QPT;
    const LayoutArgs &a;
    Slice<THREADS, QPT, NC> s1, s2;
    uint32_t x0, nb;
    size_t bbase;
    __device__ __forceinline__ TableSource(const LayoutArgs &args, uint32_t b, uint8_t *mem) : a(args)
    {
        __shared__ uint32_t s_ctl[16];
        x0 = b * S;
        s1.t = a.src_table;
        s1.nslots = a.nslots;
        s1.x0 = x0;
        s1.place(mem, a.tb, s_ctl);
        if (TWO) {
            s2.t = a.src2;
            s2.nslots = a.nslots;
            s2.x0 = x0;
            s2.place(mem + slice_index_plan(a.tb).total, a.tb, s_ctl + 8);
        }
        nb = a.B.count(b >> a.sub);
        bbase = nb ? a.B.start(b >> a.sub) : 0;
    }
    __device__ __forceinline__ void index()
    {
        __shared__ uint32_t s_w[2 * (THREADS / 32)];
        // a merge's result holds every fingerprint once whatever the tables repeat
        bool bad = s1.index(s_w, a.op != OP_MERGE);
        if (TWO) {
            __syncthreads();
            bad |= s2.index(s_w, false);
        }
        if (threadIdx.x == 0 && bad) atomicOr(a.fused_fail, 1u);
    }
    template <int NT, typename F>
    __device__ __forceinline__ void table_items(uint32_t t, F &&f) const
    {
        s1.template items<NT>(t, f);
        if (TWO) s2.template items<NT>(t, f);
    }
    template <int NT, typename F>
    __device__ __forceinline__ void batch_items(uint32_t t, F &&f) const
    {
        for_each_item<NT, NC>(a.B.items, bbase, nb, t, [&](uint32_t v) {
            const uint32_t x = (v >> SET_R) - x0;  // the batch bucket spans 2^sub layout buckets
            if (x < S) f(x, v & 31u);
        });
    }
};
template <int THREADS, int QPT>
using OneTable = TableSource<THREADS, QPT, false, false, true>;
template <int THREADS, int QPT>
using TwoTables = TableSource<THREADS, QPT, true, false, true>;
template <int THREADS, int QPT>
using LessTable = TableSource<THREADS, QPT, false, true, true>;
// the same in a launch that made the snapshot and the list itself
template <int THREADS, int QPT>
using OwnTable = TableSource<THREADS, QPT, false, false, false>;
template <int THREADS, int QPT>
using OwnLessTable = TableSource<THREADS, QPT, false, true, false>;

__host__ __device__ inline size_t set_update_smem(uint32_t tb, uint32_t threads, bool two)
{
    return set_layout_smem(tb, threads) + (two ? 2 : 1) * slice_index_plan(tb).total;
}

// One CTA per bucket, taken in ticket order so every bucket's predecessors
// are running or done when it looks back.
template <int THREADS, int QPT>
__global__ void __launch_bounds__(THREADS, (THREADS >= 1024 ? 1 : 1024 / THREADS)) k_set_layout(LayoutArgs a)
{
    if (a.a_dups && *a.a_dups) return;  // the table holds duplicates: left to k_bucket_layout
    __shared__ uint32_t s_ticket;
    if (threadIdx.x == 0) s_ticket = atomicAdd(a.ticket, 1u);
    __syncthreads();
    bucket_layout_set<THREADS, QPT, ListSource>(a, s_ticket);
}

// A build or merge that keeps every copy, or of two-byte slots.
template <int THREADS, int QPT, int BPE, bool UNIQUE>
__global__ void __launch_bounds__(THREADS, (THREADS >= 1024 ? 1 : 1024 / THREADS)) k_group_layout(LayoutArgs a)
{
    __shared__ uint32_t s_ticket;
    if (threadIdx.x == 0) s_ticket = atomicAdd(a.ticket, 1u);
    __syncthreads();
    bucket_layout_items<THREADS, QPT, GroupContents<THREADS, QPT, BPE, UNIQUE>>(a, s_ticket);
}
__host__ __device__ inline size_t group_layout_smem(uint32_t tb, uint32_t threads, uint32_t bpe, size_t cap_items)
{
    const size_t S = (size_t)1 << tb;
    return items_plan(S, threads, bpe).contents + GroupContents<32, 4, 1, false>::group_cnt_bytes(S) + cap_items * bpe;
}

// In-place merge, insert and delete: writes the live table, reads only the
// snapshot (and the second table).
enum UpdateKind : int { UPDATE_ADD = 0, UPDATE_TWO = 1, UPDATE_DEL = 2 };
template <int THREADS, int QPT, int KIND>
__global__ void __launch_bounds__(THREADS, (THREADS >= 1024 ? 1 : 768 / THREADS)) k_set_update(LayoutArgs a)
{
    __shared__ uint32_t s_ticket;
    if (threadIdx.x == 0) s_ticket = atomicAdd(a.ticket, 1u);
    __syncthreads();
    if constexpr (KIND == UPDATE_TWO) bucket_layout_set<THREADS, QPT, TwoTables>(a, s_ticket);
    else if constexpr (KIND == UPDATE_DEL) bucket_layout_set<THREADS, QPT, LessTable>(a, s_ticket);
    else bucket_layout_set<THREADS, QPT, OneTable>(a, s_ticket);
}

}  // namespace gqf

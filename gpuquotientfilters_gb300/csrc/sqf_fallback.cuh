// The general insert or delete as one cooperative launch, queued behind a
// cluster-local update and doing nothing unless that update met a stretch too
// long to walk (sqf_update.cuh, FAR_SLOTS; the table is then unchanged): the
// table's contents are extracted, the batch is bucketed, and every bucket is
// laid out again.  One launch, so that the usual empty case costs one.
#pragma once

#include "grid_sync.cuh"
#include "sqf_build.cuh"
#include "sqf_extract.cuh"

namespace gqf {

constexpr int FB_THREADS = EXTRACT_THREADS;
constexpr uint32_t FB_TB = 13;  // quotients per bucket: 32 per thread
static_assert((1u << FB_TB) == FB_THREADS * 32, "one layout CTA shape");

struct FallbackArgs {
    const uint32_t *far;
    LayoutArgs lay;  // A, B and the layout's buffers, filled below
    const uint32_t *keys;
    uint32_t n, nbytes;
    Counts3 *tiles;
    uint32_t *Q, *E, *abase, *acnt, *bcnt, *bfill, *bbase, *bitems;
    uint32_t *bar;
};

// Exclusive scan of n words by one CTA of FB_THREADS threads.
__device__ __forceinline__ void fb_scan(const uint32_t *in, uint32_t *out, uint32_t n)
{
    __shared__ uint32_t s_w[FB_THREADS / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t per = (n + FB_THREADS - 1) / FB_THREADS;
    const uint32_t i0 = min(n, tid * per), i1 = min(n, i0 + per);
    uint32_t sum = 0;
    for (uint32_t i = i0; i < i1; i++) sum += in[i];
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
    for (uint32_t i = i0; i < i1; i++) {
        out[i] = run;
        run += in[i];
    }
}

template <int BPE>
__global__ void __launch_bounds__(FB_THREADS, 2) k_update_fallback(FallbackArgs f)
{
    if (!*f.far) return;
    extern __shared__ __align__(16) uint8_t smem_layout[];
    uint32_t *s_out = reinterpret_cast<uint32_t *>(smem_layout);
    __shared__ uint32_t s_u;
    const LayoutArgs &a = f.lay;
    const uint32_t tid = threadIdx.x, gt = blockIdx.x * FB_THREADS + tid, gn = gridDim.x * FB_THREADS;
    const uint32_t ntiles = (a.nslots + EXTRACT_TILE - 1) / EXTRACT_TILE;
    const uint32_t shift = a.r + a.tb, mask = (1u << (a.q + a.r)) - 1u;
    for (uint32_t u = blockIdx.x; u < ntiles; u += gridDim.x) {
        tile_counts<BPE, false>(u, a.table, a.nslots, f.nbytes, f.tiles, nullptr);
        __syncthreads();
    }
    for (uint32_t i = gt; i < f.n; i += gn) atomicAdd(f.bcnt + ((aphash32(f.keys[i]) & mask) >> shift), 1u);
    if (!grid_sync(f.bar, a.err)) return;
    if (blockIdx.x == 0) fb_scan(f.bcnt, f.bbase, a.nb);
    if (blockIdx.x == gridDim.x - 1 && tid == 0) {  // the tiles' three counts, a few thousand
        Counts3 run{0, 0, 0};
        for (uint32_t u = 0; u < ntiles; u++) {
            const Counts3 c = f.tiles[u];
            f.tiles[u] = run;
            run.ne += c.ne;
            run.rs += c.rs;
            run.occ += c.occ;
        }
        f.tiles[ntiles] = run;
    }
    if (!grid_sync(f.bar, a.err)) return;
    for (uint32_t u = blockIdx.x; u < ntiles; u += gridDim.x) {
        occ_list<BPE, false>(u, a.table, a.nslots, f.nbytes, f.tiles, f.Q, s_out);
        __syncthreads();
    }
    for (uint32_t i = gt; i < f.n; i += gn) {
        const uint32_t fp = aphash32(f.keys[i]) & mask, b = fp >> shift;
        f.bitems[f.bbase[b] + atomicAdd(f.bfill + b, 1u)] = fp;
    }
    if (!grid_sync(f.bar, a.err)) return;
    for (uint32_t u = blockIdx.x; u < ntiles; u += gridDim.x) {
        extract<BPE, false>(u, a.table, a.nslots, f.nbytes, a.r, f.tiles, f.Q, f.E, s_out);
        __syncthreads();
    }
    if (!grid_sync(f.bar, a.err)) return;
    // bucket bounds of the extracted list; the slots past the last bucket's
    // quotients only receive spill
    const uint32_t m = f.tiles[ntiles].ne;
    auto lower = [&](uint32_t b) -> uint32_t {
        const uint64_t key = (uint64_t)b << shift;
        uint32_t lo = 0, hi = m;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if ((uint64_t)f.E[mid] < key) lo = mid + 1;
            else hi = mid;
        }
        return lo;
    };
    for (uint32_t b = gt; b < a.nb; b += gn) {
        const uint32_t lo = lower(b);
        f.abase[b] = lo;
        f.acnt[b] = lower(b + 1) - lo;
    }
    for (size_t i = ((size_t)BPE << a.q) + gt; i < f.nbytes; i += gn) a.table[i] = 0;
    if (!grid_sync(f.bar, a.err)) return;
    for (;;) {
        __syncthreads();
        if (tid == 0) s_u = atomicAdd(a.ticket, 1u);
        __syncthreads();
        const uint32_t b = s_u;
        if (b >= a.nb) break;
        bucket_layout_body<FB_THREADS, 32, BPE>(a, b);
    }
    if (!grid_sync(f.bar, a.err)) return;
    const uint32_t nf = min(*a.fix_cnt, a.fix_cap);
    for (uint32_t i = gt; i < nf; i += gn) a.table[(size_t)a.fix_list[i] * BPE + (BPE - 1)] |= 4u;
}

}  // namespace gqf

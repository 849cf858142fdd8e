// Large RSQF lookup batches through an aligned mirror of the blocks.
//
// A packed block is 57 (or 81) bytes at any alignment, so a lookup on it
// takes ten or more unaligned loads, each a separate L1 access for every lane.  A
// batch of at least one query per 16 slots first rewrites every block, once
// per call, as an aligned record (k_rsqf_mirror):
//   word 0 occupieds, 1 runEnds, 2 the offset byte, 3 + j bit plane j of the
//   remainders (bit s = bit j of slot s's remainder), padded to 32 bytes.
// A query (lookupGPU, RSQF.cu:320-399) then reads a record's first sector
// and, when its quotient is occupied, the planes: the backward walk through
// the run becomes one bit-sliced comparison of all 64 slots.  The records are
// the table's own fields, so every table gives the direct lookup's answers.
//
// Bounds: L1 accesses, two or three 32-byte sectors a query.
#pragma once

#include "rsqf.cuh"

namespace GQF_RSQF_NS {

constexpr uint32_t RMIR_WORDS = (3 + RSQF_R + 3) / 4 * 4;  // 8 for 5-bit remainders, 12 for 8-bit
constexpr int RMIR_THREADS = 128;                         // blocks per build CTA
__host__ __device__ inline size_t rmir_bytes(uint32_t nblocks) { return (size_t)(nblocks + 1) * RMIR_WORDS * 8; }

__device__ __forceinline__ void ld_sector(const uint64_t *p, uint64_t (&w)[4])
{
    asm volatile("ld.global.nc.v4.u64 {%0,%1,%2,%3}, [%4];" : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3]) : "l"(p));
}
__device__ __forceinline__ void st_sector(uint64_t *p, const uint64_t *w)
{
    asm volatile("st.global.v4.u64 [%0], {%1,%2,%3,%4};" ::"l"(p), "l"(w[0]), "l"(w[1]), "l"(w[2]), "l"(w[3]) : "memory");
}

// One thread per block; the CTA's packed blocks are staged in shared memory
// with coalesced 16-byte loads (128 blocks are a multiple of 16 bytes; the
// table is 16-byte aligned and ends with 16 spare bytes).
static __global__ void __launch_bounds__(RMIR_THREADS) k_rsqf_mirror(const uint8_t *__restrict__ t, uint32_t nblocks,
                                                                     uint64_t *__restrict__ rec)
{
    constexpr uint32_t BYTES = RMIR_THREADS * RSQF_BB;
    static_assert(BYTES % 16 == 0, "whole 16-byte words per CTA");
    __shared__ __align__(16) uint32_t s_raw[BYTES / 4 + 4];
    const size_t total = (size_t)(nblocks + 1) * RSQF_BB, c0 = (size_t)blockIdx.x * BYTES;
    for (uint32_t i = threadIdx.x * 16; i < BYTES; i += RMIR_THREADS * 16) {
        uint4 v = make_uint4(0, 0, 0, 0);
        if (c0 + i < total) v = __ldg(reinterpret_cast<const uint4 *>(t + c0 + i));  // within the spare bytes at the end
        *reinterpret_cast<uint4 *>(reinterpret_cast<uint8_t *>(s_raw) + i) = v;
    }
    if (threadIdx.x < 4) s_raw[BYTES / 4 + threadIdx.x] = 0;
    __syncthreads();
    const uint32_t b = blockIdx.x * RMIR_THREADS + threadIdx.x;
    if (b > nblocks) return;
    const uint32_t o = threadIdx.x * RSQF_BB;
    auto u32_at = [&](uint32_t byte) -> uint32_t {
        const uint32_t w = byte >> 2;
        return __funnelshift_r(s_raw[w], s_raw[w + 1], 8 * (byte & 3u));
    };
    uint64_t out[RMIR_WORDS];
#pragma unroll
    for (uint32_t k = 0; k < RMIR_WORDS; k++) out[k] = 0;
    out[0] = u32_at(o + 1) | ((uint64_t)u32_at(o + 5) << 32);
    out[1] = u32_at(o + 9) | ((uint64_t)u32_at(o + 13) << 32);
    out[2] = u32_at(o) & 0xFFu;
    // bit planes, 32 slots (RSQF_R words) at a time
#pragma unroll
    for (uint32_t h = 0; h < 2; h++) {
        uint32_t pl[RSQF_R];
#pragma unroll
        for (uint32_t j = 0; j < RSQF_R; j++) pl[j] = 0;
        uint32_t w[RSQF_R + 1];
#pragma unroll
        for (uint32_t k = 0; k < RSQF_R; k++) w[k] = u32_at(o + 17 + 4 * (h * RSQF_R + k));
        w[RSQF_R] = 0;
#pragma unroll
        for (uint32_t s = 0; s < 32; s++) {
            const uint32_t bit = s * RSQF_R, f = __funnelshift_r(w[bit >> 5], w[(bit >> 5) + 1], bit & 31u);
#pragma unroll
            for (uint32_t j = 0; j < RSQF_R; j++) pl[j] |= ((f >> j) & 1u) << s;
        }
#pragma unroll
        for (uint32_t j = 0; j < RSQF_R; j++) out[3 + j] |= (uint64_t)pl[j] << (32 * h);
    }
    uint64_t *d = rec + (size_t)b * RMIR_WORDS;
#pragma unroll
    for (uint32_t k = 0; k < RMIR_WORDS; k += 4) st_sector(d + k, out + k);
}

// rsqf_lookup on the mirror.
__device__ __forceinline__ int32_t rsqf_lookup_mirror(const uint64_t *__restrict__ rec, uint32_t nblocks, uint32_t q,
                                                      uint32_t fp)
{
    const uint32_t fq = (fp >> RSQF_R) & ((1u << q) - 1u), fr = fp & RSQF_RMASK;
    const uint32_t home = fq / RSQF_SPB, sl = fq % RSQF_SPB;
    uint32_t b = home;
    uint64_t s0[4];
    ld_sector(rec + (size_t)b * RMIR_WORDS, s0);
    if (!((s0[0] >> sl) & 1ull)) return -1;
    uint32_t rank = rank64(s0[0], sl), off = (uint32_t)s0[2];
    uint64_t m = s0[1] & ~lowmask64(off);
    for (uint32_t c = (uint32_t)__popcll(m); rank > c; c = (uint32_t)__popcll(m)) {
        rank -= c;
        off = off > RSQF_SPB ? off - RSQF_SPB : 0u;
        if (++b > nblocks) return -1;
        ld_sector(rec + (size_t)b * RMIR_WORDS, s0);
        m = s0[1] & ~lowmask64(off);
    }
    // the rank-th run end of m
    const uint32_t clo = (uint32_t)__popc((uint32_t)m);
    uint32_t hi = rank > clo ? 32 + nth_bit((uint32_t)(m >> 32), (int)(rank - clo - 1))
                             : nth_bit((uint32_t)m, (int)rank - 1);
    // down through the run: the first slot with a remainder <= fr decides.
    // The run goes down to the slot above the next lower run end, no lower
    // than fq; its last slot is looked at in any case.
    uint64_t first = 1ull << hi;
    for (;;) {
        const uint64_t below = s0[1] & (first ? lowmask64(hi) : lowmask64(hi + 1));
        uint32_t lo = below ? 64u - (uint32_t)__clzll((long long)below) : 0u;
        const bool goes_on = lo == 0;
        if (b == home) lo = max(lo, sl);
        const uint64_t run = first | (lowmask64(hi + 1) & ~lowmask64(lo));
        uint64_t eq = ~0ull, gt = 0ull;
        uint64_t pl[RMIR_WORDS - 4];
        ld_sector(rec + (size_t)b * RMIR_WORDS + 4, *reinterpret_cast<uint64_t(*)[4]>(pl));
        if constexpr (RMIR_WORDS > 8)
            ld_sector(rec + (size_t)b * RMIR_WORDS + 8, *reinterpret_cast<uint64_t(*)[4]>(pl + 4));
#pragma unroll
        for (int j = (int)RSQF_R - 1; j >= 0; j--) {
            const uint64_t P = j ? pl[j - 1] : s0[3], fb = 0ull - (uint64_t)((fr >> j) & 1u);
            gt |= eq & P & ~fb;
            eq &= ~(P ^ fb);
        }
        const uint64_t cand = ~gt & run;
        if (cand) {
            const uint32_t s = 63u - (uint32_t)__clzll((long long)cand);
            return ((eq >> s) & 1ull) ? (int32_t)(b * RSQF_SPB + s) : -1;
        }
        if (!goes_on || b <= home) return -1;
        b--;
        ld_sector(rec + (size_t)b * RMIR_WORDS, s0);
        hi = 63;
        first = 0;
    }
}

constexpr int RMIR_LOOKUP_THREADS = 256;
static __global__ void __launch_bounds__(RMIR_LOOKUP_THREADS) k_rsqf_lookup_mirror(const uint32_t *__restrict__ keys,
                                                                                  uint32_t n,
                                                                                  const uint64_t *__restrict__ rec,
                                                                                  uint32_t nblocks, uint32_t q,
                                                                                  int32_t *__restrict__ out)
{
    const uint32_t mask = (1u << (q + RSQF_R)) - 1u;
    for (uint32_t i = blockIdx.x * RMIR_LOOKUP_THREADS + threadIdx.x; i < n; i += gridDim.x * RMIR_LOOKUP_THREADS)
        out[i] = rsqf_lookup_mirror(rec, nblocks, q, aphash32(__ldg(keys + i)) & mask);
}

}  // namespace GQF_RSQF_NS

// Cluster-local inserts and deletes: only the slots that change are touched.
//
// The reference applies updates in rounds of one insert or delete per
// supercluster, each a sequential shift (quotientFilter.cu:407-634,
// :1060-1297).  Here a batch is first resolved against the unchanged table,
// and then every independent stretch of slots is rewritten by one thread:
//
//   delete  k_del_locate  each key claims one stored copy of its fingerprint
//                         and, once per unit, the unit the copy lies in.
//           k_del_apply   one thread per claimed unit moves the unit's kept
//                         elements left.
//   insert  k_ins_stage   drops keys already stored or repeated in the batch
//                         and groups the rest by quotient range.
//           k_ins_sort    sorts each group and finds, per key, the slot it
//                         goes in front of and the empty slot its shift ends in.
//           k_ins_groups  marks the clusters that an earlier cluster's
//                         inserts spill into.
//           k_ins_apply   one thread per group of connected clusters moves
//                         its elements right and puts the new ones in.
//
// A unit is a stretch from an unshifted element up to the next unshifted or
// empty slot.  An unshifted element cannot move left, so a delete changes
// nothing outside its unit, and the unit's first run is its first slot's
// quotient.  A cluster is a stretch between empty slots; an insert moves the
// elements from its place to the next empty slot, and only when a cluster
// gets more inserts than the empty slot after it can take does it reach the
// next one.  Both hold for every table, with or without repeated
// fingerprints; the results are the canonical table, as the reference's.
//
// Bounds: random 32-byte sectors, about four per key, and the longest
// stretch's serial walk.  Rewriting the table bucket by bucket cost its whole
// length whatever the batch.
#pragma once

#include "sqf_lookup.cuh"

namespace gqf {

constexpr int UPD_THREADS = 256;
constexpr uint32_t UPD_NONE = 0xFFFFFFFFu;
// A stretch longer than this (a nearly full table) is not walked: the kernel
// that meets it sets *far, nothing has been changed yet, the apply kernels do
// nothing, and k_update_fallback rebuilds the table.
constexpr uint32_t FAR_SLOTS = 5120;  // more than the slots of q = 12

// Slots of the live table: element i = rem << 3 | occupied << 2 |
// continuation << 1 | shifted.
template <int BPE>
struct SlotTable {
    uint8_t *t;
    uint32_t nslots;
    __device__ __forceinline__ uint32_t get(uint32_t i) const
    {
        if (BPE == 1) return t[i];
        const uint32_t v = reinterpret_cast<const uint16_t *>(t)[i];
        return ((v & 0xFFu) << 8) | (v >> 8);
    }
    __device__ __forceinline__ void put(uint32_t i, uint32_t e) const
    {
        if (BPE == 1) t[i] = (uint8_t)e;
        else reinterpret_cast<uint16_t *>(t)[i] = (uint16_t)(((e & 0xFFu) << 8) | (e >> 8));
    }
    // first empty slot at or after i (nslots: none; UPD_NONE: too far)
    __device__ __forceinline__ uint32_t next_empty(uint32_t i) const
    {
        const uint32_t end = i + FAR_SLOTS;
        if (BPE == 1) {
            while (i < nslots) {
                if (i > end) return UPD_NONE;
                const uint32_t w = i >> 3;
                if (8 * w + 8 > nslots) break;  // the ragged last word slot by slot
                const uint64_t x = reinterpret_cast<const unsigned long long *>(t)[w];
                const uint64_t em = ~(x | (x >> 1) | (x >> 2)) & BL_LO & ~bytes_below(i & 7u);
                if (em) return 8 * w + lowest_byte(em);
                i = 8 * w + 8;
            }
        }
        while (i < nslots && (get(i) & 7u)) {
            if (i++ > end) return UPD_NONE;
        }
        return i;
    }
};

// Where quotient fq's run is or would go, from the unchanged table.
//   unit: the last unshifted slot at or below fq (the start of fq's unit when
//         fq is occupied);
//   occ:  fq has a run;
//   pos:  occ: the run's first slot; otherwise the slot a first element of fq
//         goes in front of (the next run's start or the first empty slot);
//   far:  the walk went past FAR_SLOTS, pos is not known.
struct RunPlace {
    uint32_t unit, pos;
    bool occ, far;
};
template <int BPE>
__device__ __forceinline__ RunPlace find_run(const SlotTable<BPE> &v, uint32_t fq)
{
    RunPlace r;
    r.far = false;
    r.pos = v.nslots;
    int D = 0;  // runs of lower quotients starting at or after fq
    uint32_t b = fq;
    if (BPE == 1) {
        constexpr uint64_t OCC = 0x0404040404040404ull;
        const unsigned long long *t64 = reinterpret_cast<const unsigned long long *>(v.t);
        const uint32_t w = fq >> 3, k = fq & 7u;  // quotients lie in whole words (2^q >= 128 slots)
        const uint64_t x = t64[w];
        r.occ = (x >> (8 * k + 2)) & 1u;
        uint64_t st = bl_unshifted(x) & bytes_below(k + 1);
        uint64_t y = x, in = bytes_below(k);
        uint32_t ww = w;
        while (!st) {
            D += popc64(y & OCC & in) - popc64(bl_run_starts(y) & in);
            if (ww == 0) break;
            if (w - ww > FAR_SLOTS / 8) {
                r.far = true;
                return r;
            }
            y = t64[--ww];
            in = ~0ull;
            st = bl_unshifted(y);
        }
        const uint32_t hb = st ? highest_byte(st) : 0u;
        if (st) {
            const uint64_t R = in & ~bytes_below(hb);
            D += popc64(y & OCC & R) - popc64(bl_run_starts(y) & R);
        }
        r.unit = 8 * ww + hb;
        // forward: the (D+1)-th run start at or after fq; without a run of
        // fq, no further than the first empty slot
        uint64_t from = ~bytes_below(k), z = x;
        uint32_t wz = w;
        for (;;) {
            const uint64_t rs = bl_run_starts(z) & from;
            const uint64_t em = ~(z | (z >> 1) | (z >> 2)) & BL_LO & from;
            const int c = popc64(rs);
            uint32_t at = 8;
            if (c > max(D, 0)) {
                uint64_t m = rs;
                for (int i = 0; i < D; i++) m &= m - 1;
                at = lowest_byte(m);
            }
            if (!r.occ && em) at = min(at, lowest_byte(em));
            if (at < 8) {
                r.pos = 8 * wz + at;
                return r;
            }
            D -= c;
            wz++;
            if (8 * wz + 8 > v.nslots) break;
            if (wz - w > FAR_SLOTS / 8) {
                r.far = true;
                return r;
            }
            z = t64[wz];
            from = ~0ull;
        }
        // the ragged last word
        for (uint32_t s = 8 * wz; s < v.nslots; s++) {
            const uint32_t e = v.get(s);
            if (!(e & 7u) ? !r.occ : (!(e & 2u) && D-- == 0)) {
                r.pos = s;
                return r;
            }
        }
        return r;
    }
    r.occ = (v.get(fq) >> 2) & 1u;
    while (b > 0) {
        if (!(v.get(b) & 1u)) break;
        if (fq - b > FAR_SLOTS) {
            r.far = true;
            return r;
        }
        b--;
        const uint32_t e = v.get(b);
        D += (int)((e >> 2) & 1u) - (int)((e & 7u) && !(e & 2u));
    }
    r.unit = b;
    for (uint32_t s = fq; s < v.nslots; s++) {
        const uint32_t e = v.get(s);
        if (!(e & 7u) ? !r.occ : (!(e & 2u) && D-- == 0)) {
            r.pos = s;
            return r;
        }
        if (s - fq > FAR_SLOTS) {
            r.far = true;
            return r;
        }
    }
    return r;
}

// ------------------------------------------------------------------ delete
// claim: two bits per slot, bit 0 "delete the element here", bit 1 "a thread
// has this unit" (at the unit's first slot).  lead[i] = the unit key i leads,
// or UPD_NONE.
template <int BPE>
__global__ void __launch_bounds__(UPD_THREADS) k_del_locate(const uint32_t *__restrict__ keys, uint32_t n,
                                                           SlotTable<BPE> v, uint32_t q, uint32_t r,
                                                           uint32_t *__restrict__ claim, uint32_t *__restrict__ lead,
                                                           uint32_t *far)
{
    const uint32_t i = blockIdx.x * UPD_THREADS + threadIdx.x;
    if (i >= n) return;
    const uint32_t fp = aphash32(__ldg(keys + i)) & ((1u << (q + r)) - 1u);
    const uint32_t fq = fp >> r, fr = fp & ((1u << r) - 1u);
    uint32_t mine = UPD_NONE;
    if ((v.get(fq) >> 2) & 1u) {
        const RunPlace p = find_run<BPE>(v, fq);
        if (p.far) *far = 1;
        for (uint32_t s = p.pos; s < v.nslots && !p.far; s++) {
            const uint32_t e = v.get(s);
            if (s > p.pos && !(e & 2u)) break;  // end of the run
            const uint32_t rem = e >> 3;
            if (rem > fr) break;
            if (rem < fr) continue;
            // one copy per occurrence: the first copy nobody claimed
            const uint32_t bit = 1u << (2 * (s & 15u));
            if (!(atomicOr(claim + (s >> 4), bit) & bit)) {
                const uint32_t ub = 2u << (2 * (p.unit & 15u));
                if (!(atomicOr(claim + (p.unit >> 4), ub) & ub)) {
                    mine = p.unit;
                    uint32_t e1 = s + 1;  // the unit's end
                    while (e1 < v.nslots && (v.get(e1) & 1u) && e1 - mine <= FAR_SLOTS) e1++;
                    if (e1 - mine > FAR_SLOTS) *far = 1;
                }
                break;
            }
        }
    }
    lead[i] = mine;
}

// Rewrites each led unit without its claimed elements.  Every kept element
// goes to max(its quotient, the slot after the one before it).
template <int BPE>
__global__ void __launch_bounds__(UPD_THREADS) k_del_apply(uint32_t n, SlotTable<BPE> v,
                                                          const uint32_t *__restrict__ claim,
                                                          const uint32_t *__restrict__ lead,
                                                          const uint32_t *__restrict__ far)
{
    const uint32_t i = blockIdx.x * UPD_THREADS + threadIdx.x;
    if (i >= n || *far) return;
    const uint32_t u = lead[i];
    if (u == UPD_NONE) return;
    uint32_t quot = u;  // quotient of the current run
    uint32_t c = u;     // first free slot
    uint32_t kept = 0;  // elements kept of the current run
    uint32_t cw = UPD_NONE, cbits = 0;
    uint32_t t = u;
    for (; t < v.nslots; t++) {
        const uint32_t e = v.get(t);
        if (t > u && !(e & 1u)) break;  // the next unit, or an empty slot
        if (t > u && !(e & 2u)) {       // a new run
            if (!kept) v.put(quot, v.get(quot) & ~4u);
            do quot++;
            while (quot < t && !(v.get(quot) & 4u));
            kept = 0;
        }
        if ((t >> 4) != cw) {
            cw = t >> 4;
            cbits = claim[cw];
        }
        if ((cbits >> (2 * (t & 15u))) & 1u) continue;
        for (; c < quot; c++) v.put(c, 0u);
        const uint32_t ne = (e & ~7u) | (kept ? 2u : 0u) | (c != quot ? 1u : 0u);
        if (c != t || ne != (e & ~4u)) v.put(c, ne | (v.get(c) & 4u));
        c++;
        kept++;
    }
    if (!kept) v.put(quot, v.get(quot) & ~4u);
    for (; c < t; c++) v.put(c, 0u);
}

// ------------------------------------------------------------------ insert
// The batch's new fingerprints: bucket b (quotient range fp >> shift) holds
// cnt[b] of them from base[b], sorted by k_ins_sort.
//   ip[k]  slot the key goes in front of; INS_HEAD: in front of its run's
//          first element, or first of a new run
//   gap[k] first empty slot at or after its quotient; INS_NEWQ: its quotient
//          has no run yet; INS_COVERED (first key of a gap): an earlier
//          gap's inserts reach this one's cluster
constexpr uint32_t INS_HEAD = 1u << 31, INS_COVERED = 1u << 31, INS_NEWQ = 1u << 30;
constexpr uint32_t INS_GAP = INS_NEWQ - 1;

struct InsBatch {
    uint32_t nb, shift, stride, hmask;
    uint32_t *cnt, *base;            // per bucket
    uint32_t *n_over, *pool;         // keys past their bucket's stride; pool space handed out
    uint32_t *fp, *ip, *gap;         // nb * stride entries, then the pool of n
    uint32_t *over;                  // n
    uint32_t *seen;                  // hash set of hmask + 1 entries, all ones
};

template <int BPE>
__global__ void __launch_bounds__(UPD_THREADS) k_ins_stage(const uint32_t *__restrict__ keys, uint32_t n,
                                                          SlotTable<BPE> v, uint32_t q, uint32_t r, InsBatch b,
                                                          uint32_t *far)
{
    const uint32_t i = blockIdx.x * UPD_THREADS + threadIdx.x;
    if (i >= n) return;
    const uint32_t fp = aphash32(__ldg(keys + i)) & ((1u << (q + r)) - 1u);
    // repeated in the batch: only the thread whose entry this is goes on
    uint32_t h = (fp * 0x9E3779B1u) >> 7;
    for (uint32_t tries = 0; tries <= b.hmask; tries++, h++) {
        uint32_t *slot = b.seen + (h & b.hmask);
        uint32_t cur = *reinterpret_cast<volatile uint32_t *>(slot);
        if (cur == UPD_NONE) cur = atomicCAS(slot, UPD_NONE, fp);
        if (cur == UPD_NONE) break;
        if (cur == fp) return;
    }
    const uint32_t fq = fp >> r, fr = fp & ((1u << r) - 1u);
    if ((v.get(fq) >> 2) & 1u) {
        const RunPlace p = find_run<BPE>(v, fq);
        if (p.far) *far = 1;
        for (uint32_t s = p.pos; s < v.nslots && !p.far; s++) {
            const uint32_t e = v.get(s);
            if (s > p.pos && !(e & 2u)) break;
            const uint32_t rem = e >> 3;
            if (rem == fr) return;  // stored already
            if (rem > fr) break;
        }
    }
    const uint32_t bk = fp >> b.shift, k = atomicAdd(b.cnt + bk, 1u);
    if (k < b.stride) b.fp[(size_t)bk * b.stride + k] = fp;
    else b.over[atomicAdd(b.n_over, 1u)] = fp;
}

// Ascending sort of m words by the CTA (all comparators ascending, so the
// missing tail of the last power of two acts as the largest values).
template <int THREADS>
__device__ __forceinline__ void cta_sort(uint32_t *a, uint32_t m)
{
    uint32_t p2 = 1;
    while (p2 < m) p2 <<= 1;
    for (uint32_t k = 2; k <= p2; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            const bool flip = j == (k >> 1);
            for (uint32_t i = threadIdx.x; i < p2 / 2; i += THREADS) {
                const uint32_t lo = (i / j) * 2 * j + (i % j), hi = flip ? (lo ^ (k - 1)) : lo + j;
                if (hi < m) {
                    const uint32_t x = a[lo], y = a[hi];
                    if (x > y) {
                        a[lo] = y;
                        a[hi] = x;
                    }
                }
            }
            __syncthreads();
        }
    }
}

constexpr int INS_THREADS = 128;
constexpr uint32_t INS_SMEM_KEYS = 2048;

template <int BPE>
__global__ void __launch_bounds__(INS_THREADS) k_ins_sort(SlotTable<BPE> v, uint32_t r, InsBatch b, uint32_t *far)
{
    __shared__ uint32_t s_key[INS_SMEM_KEYS];
    __shared__ uint32_t s_n, s_base;
    const uint32_t bk = blockIdx.x, cnt = b.cnt[bk], tid = threadIdx.x;
    uint32_t base = bk * b.stride;
    const uint32_t direct = min(cnt, b.stride);
    uint32_t *key = s_key;
    if (cnt > INS_SMEM_KEYS) {  // sorted in place in the pool
        if (tid == 0) s_base = b.nb * b.stride + atomicAdd(b.pool, cnt);
        __syncthreads();
        key = b.fp + s_base;
    }
    for (uint32_t i = tid; i < direct; i += INS_THREADS) key[i] = b.fp[base + i];
    if (cnt > b.stride) {  // the rest is among the keys that overflowed
        if (cnt <= INS_SMEM_KEYS && tid == 0) s_base = b.nb * b.stride + atomicAdd(b.pool, cnt);
        if (tid == 0) s_n = direct;
        __syncthreads();
        base = s_base;
        const uint32_t no = *b.n_over;
        for (uint32_t i = tid; i < no; i += INS_THREADS) {
            const uint32_t fp = b.over[i];
            if ((fp >> b.shift) == bk) key[atomicAdd(&s_n, 1u)] = fp;
        }
    }
    __syncthreads();
    if (tid == 0) b.base[bk] = base;
    cta_sort<INS_THREADS>(key, cnt);
    for (uint32_t i = tid; i < cnt; i += INS_THREADS) {
        const uint32_t fp = key[i], fq = fp >> r, fr = fp & ((1u << r) - 1u);
        const RunPlace p = find_run<BPE>(v, fq);
        uint32_t ip = p.pos, head = INS_HEAD;
        if (p.occ && !p.far) {
            for (; ip < v.nslots; ip++) {
                const uint32_t e = v.get(ip);
                if (ip > p.pos && !(e & 2u)) break;  // end of the run
                if ((e >> 3) > fr) break;
            }
            if (ip != p.pos) head = 0;
        }
        const uint32_t gap = p.far ? UPD_NONE : v.next_empty(ip);
        if (gap == UPD_NONE) *far = 1;
        b.fp[base + i] = fp;
        b.ip[base + i] = ip | head;
        b.gap[base + i] = (gap & INS_GAP) | (p.occ ? 0u : INS_NEWQ);
    }
}

// Walks the sorted keys of all buckets in order.
struct InsPos {
    uint32_t bk, i;
};
__device__ __forceinline__ bool ins_valid(const InsBatch &b, InsPos k) { return k.bk < b.nb; }
__device__ __forceinline__ uint32_t ins_at(const InsBatch &b, InsPos k) { return b.base[k.bk] + k.i; }
__device__ __forceinline__ InsPos ins_next(const InsBatch &b, InsPos k)
{
    if (++k.i < b.cnt[k.bk]) return k;
    k.i = 0;
    do k.bk++;
    while (k.bk < b.nb && !b.cnt[k.bk]);
    return k;
}
// false: k is the first key
__device__ __forceinline__ bool ins_prev(const InsBatch &b, InsPos &k)
{
    if (k.i) {
        k.i--;
        return true;
    }
    while (k.bk > 0) {
        const uint32_t c = b.cnt[--k.bk];
        if (c) {
            k.i = c - 1;
            return true;
        }
    }
    return false;
}
// the first key of its gap
__device__ __forceinline__ bool ins_first(const InsBatch &b, InsPos k)
{
    const uint32_t g = b.gap[ins_at(b, k)] & INS_GAP;
    InsPos p = k;
    return !ins_prev(b, p) || (b.gap[ins_at(b, p)] & INS_GAP) != g;
}
// From the first key k of gap g: takes the keys of one gap after the other
// until their empty slots have taken every shift.  Returns the last gap
// (nslots: the table is full), the last key taken in `last`; mark(key) for
// the first key of every gap after the first.
template <int BPE, typename Mark>
__device__ __forceinline__ uint32_t ins_walk(const InsBatch &b, const SlotTable<BPE> &v, InsPos k, InsPos &last,
                                             Mark &&mark)
{
    uint32_t pending = 0, g = b.gap[ins_at(b, k)] & INS_GAP;
    const uint32_t g0 = g;
    for (;;) {
        if (g != g0 && ins_valid(b, k) && (b.gap[ins_at(b, k)] & INS_GAP) == g && !mark(ins_at(b, k))) return g;
        while (ins_valid(b, k) && (b.gap[ins_at(b, k)] & INS_GAP) == g) {
            pending++;
            last = k;
            k = ins_next(b, k);
        }
        if (g >= v.nslots || --pending == 0) return g;
        g = v.next_empty(g + 1);
        if (g - g0 > FAR_SLOTS) return g == v.nslots ? g : UPD_NONE;
    }
}

template <int BPE>
__global__ void __launch_bounds__(INS_THREADS) k_ins_groups(SlotTable<BPE> v, InsBatch b, uint32_t *far)
{
    if (*reinterpret_cast<volatile uint32_t *>(far)) return;
    const uint32_t bk = blockIdx.x, cnt = b.cnt[bk];
    for (uint32_t i = threadIdx.x; i < cnt; i += INS_THREADS) {
        const InsPos k{bk, i};
        if (!ins_first(b, k)) continue;
        InsPos last;
        // a walker whose own start is covered leaves the rest to the walker
        // that covered it, whose shifts reach at least as far
        const volatile uint32_t *own = b.gap + ins_at(b, k);
        if (ins_walk<BPE>(b, v, k, last, [&](uint32_t at) {
                atomicOr(b.gap + at, INS_COVERED);
                return !(*own & INS_COVERED);
            }) == UPD_NONE)
            *far = 1;
    }
}

template <int BPE>
__global__ void __launch_bounds__(INS_THREADS) k_ins_apply(SlotTable<BPE> v, uint32_t r, InsBatch b, uint32_t *err,
                                                          const uint32_t *__restrict__ far)
{
    if (*far) return;
    const uint32_t bk = blockIdx.x, cnt = b.cnt[bk];
    for (uint32_t i = threadIdx.x; i < cnt; i += INS_THREADS) {
        InsPos k{bk, i};
        if ((b.gap[ins_at(b, k)] & INS_COVERED) || !ins_first(b, k)) continue;
        InsPos last;
        const uint32_t g = ins_walk<BPE>(b, v, k, last, [](uint32_t) { return true; });
        if (g >= v.nslots) {
            atomicOr(err, DEV_ERR_FULL);
            continue;
        }
        // right to left from the last empty slot: d = slots an element here moves
        k = last;
        uint32_t at = ins_at(b, k), ipk = b.ip[at];
        uint32_t d = 0;
        for (uint32_t s = g;; s--) {
            const uint32_t e = v.get(s);
            const bool here = (ipk & ~INS_HEAD) == s;
            if (!(e & 7u)) {
                d++;  // an empty slot takes one shift
            } else {
                // the old head of a run continues it when a new key goes in front
                const uint32_t cont = (here && (ipk & INS_HEAD) && !(b.gap[at] & INS_NEWQ)) ? 2u : 0u;
                v.put(s + d, (e & ~4u) | 1u | cont | (v.get(s + d) & 4u));
            }
            while ((ipk & ~INS_HEAD) == s) {
                const uint32_t fp = b.fp[at], fq = fp >> r, pos = s + d - 1;
                const bool newq = (b.gap[at] & INS_NEWQ) != 0, head = (ipk & INS_HEAD) != 0;
                d--;
                bool behind = false;  // a smaller new key of the same quotient
                const bool more = ins_prev(b, k);
                if (more) {
                    at = ins_at(b, k);
                    behind = (b.fp[at] >> r) == fq;
                    ipk = b.ip[at];
                }
                v.put(pos, ((fp & ((1u << r) - 1u)) << 3) | ((head && !behind) ? 0u : 2u) | (pos != fq ? 1u : 0u) |
                               (v.get(pos) & 4u));
                if (newq && !behind) v.put(fq, v.get(fq) | 4u);
                if (!d || !more) break;
            }
            if (!d) break;
        }
    }
}

}  // namespace gqf

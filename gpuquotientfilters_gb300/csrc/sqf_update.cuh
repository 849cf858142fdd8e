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
//                         elements left (k_del_units: units with several).
//   insert  k_ins_stage   drops keys already stored or repeated in the batch
//                         and groups the rest by quotient range.
//           k_ins_sort    sorts each group and finds, per key, the slot it
//                         goes in front of and the empty slot its shift ends in.
//           k_ins_groups  marks the clusters that an earlier cluster's
//                         inserts spill into.
//           k_ins_apply   one thread per group of connected clusters moves
//                         its elements right and puts the new ones in
//                         (k_ins_lists: groups of several keys).
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

#include "sqf_walk.cuh"

namespace gqf {

constexpr int UPD_THREADS = 256;
constexpr uint32_t UPD_NONE = WALK_NONE;
// Single shifts of one-byte slots, a word (8 slots) at a time.  Only the
// slots of the thread's own stretch change; they are written as XOR
// differences, so a word shared with a neighbour's stretch needs no care.
// Not used in the table's ragged last word.
__device__ __forceinline__ uint64_t ldw(const SlotTable<1> &v, uint32_t w)
{
    return __ldcg(reinterpret_cast<const unsigned long long *>(v.t) + w);
}
__device__ __forceinline__ void xorw(const SlotTable<1> &v, uint32_t w, uint64_t diff)
{
    if (diff) atomicXor(reinterpret_cast<unsigned long long *>(v.t) + w, (unsigned long long)diff);
}
constexpr uint64_t OCC8 = 0x0404040404040404ull;
// bytes [a, b) of a word, a and b clamped to it (slots relative to the word)
__device__ __forceinline__ uint64_t bytes_range(int a, int b)
{
    return bytes_below((uint32_t)min(max(b, 0), 8)) & ~bytes_below((uint32_t)min(max(a, 0), 8));
}

// Removes the element at slot s (quotient fq) of the stretch that runs to
// before slot `end`: everything behind it moves one slot left.  A run start
// moving to its quotient's own slot becomes unshifted: slot y's new element
// comes from y + 1, and is at home when it starts a run, quotient y is
// occupied, and only one run (y's) was pending at y + 1.  D: runs pending at
// s + 1, the quotients above fq occupied up to s.
__device__ __forceinline__ void shift_left(const SlotTable<1> &v, uint32_t s, uint32_t end, uint32_t fq, uint32_t D)
{
    uint32_t w = s >> 3;
    uint64_t x = ldw(v, w);
    const uint32_t es = (uint32_t)(x >> (8 * (s & 7u))) & 0xFFu;
    bool emptied = false;
    for (const uint32_t w0 = w;; w++) {
        const int b0 = (int)(8 * w);
        const uint64_t nx = 8 * w + 8 < end ? ldw(v, w + 1) : 0ull;
        const uint64_t src = (x >> 8) | (nx << 56);
        const uint64_t cnt_in = w == w0 ? bytes_range((int)(s + 1) - b0, 8) : ~0ull;
        const uint64_t oc = (x >> 2) & BL_LO, po = (oc & cnt_in) * BL_LO, pr = (bl_run_starts(x) & cnt_in) * BL_LO;
        const uint64_t d1 = ((uint64_t)min(D, 120u) * BL_LO + po - pr) ^ BL_LO;       // 0: one run pending
        const uint64_t one = ~((d1 | ((d1 & ~BL_HI) + ~BL_HI)) >> 7) & BL_LO;         // its zero bytes
        const uint64_t home = bl_run_starts(src) & oc & one;
        uint64_t nw = (src & ~(OCC8 | BL_LO)) | (x & OCC8) | (BL_LO & ~home);
        if (w == w0) {
            const uint32_t sh = 8 * (s & 7u);
            const uint32_t ns = (uint32_t)(src >> sh) & 0xFFu;
            if (!(es & 2u)) {  // the head of its run goes
                if (s + 1 < end && (ns & 2u)) {  // the next element heads it, where the old head was
                    nw = (nw & ~(0xFFull << sh)) | ((uint64_t)((ns & ~7u) | (es & 5u)) << sh);
                } else {
                    emptied = true;
                }
            }
        }
        const uint64_t mine = bytes_range((int)s - b0, (int)(end - 1) - b0);
        const uint64_t last = bytes_range((int)(end - 1) - b0, (int)end - b0);  // the slot left over
        uint64_t diff = ((nw ^ x) & mine) | (x & ~OCC8 & last);
        if (w == w0 && emptied && (fq >> 3) == w) {
            diff ^= 4ull << (8 * (fq & 7u));
            emptied = false;
        }
        xorw(v, w, diff);
        D += (uint32_t)popc64(oc & cnt_in) - (uint32_t)popc64(bl_run_starts(x) & cnt_in);
        if (8 * w + 8 >= end) break;
        x = nx;
    }
    if (emptied) xorw(v, fq >> 3, 4ull << (8 * (fq & 7u)));
}

// Puts element e (its byte without the occupied bit) into slot s, moving the
// elements from s up to before the empty slot g one slot right; `cont`: the
// element at s becomes a continuation.
__device__ __forceinline__ void shift_right(const SlotTable<1> &v, uint32_t s, uint32_t g, uint32_t e, bool cont)
{
    uint64_t px = 0;  // the word before
    for (uint32_t w = s >> 3; w <= (g >> 3); w++) {
        const int b0 = (int)(8 * w);
        const uint64_t x = ldw(v, w);
        uint64_t nw = (((x << 8) | (px >> 56)) & ~(OCC8 | BL_LO)) | BL_LO;
        if (cont && s + 1 >= 8 * w && s + 1 < 8 * w + 8) nw |= 2ull << (8 * ((s + 1) & 7u));
        if ((s >> 3) == w) nw = (nw & ~(0xFFull << (8 * (s & 7u)))) | ((uint64_t)e << (8 * (s & 7u)));
        xorw(v, w, (nw ^ x) & ~OCC8 & bytes_range((int)s - b0, (int)(g + 1) - b0));
        px = x;
    }
}

// Changes the bits `diff` of slot i's element (a word of 4 slot bytes inside
// the table; k_del_units and k_ins_lists use this size only, the apply kernels
// 8-byte words only).
template <int BPE>
__device__ __forceinline__ void xor_slot(const SlotTable<BPE> &v, uint32_t i, uint32_t diff)
{
    if (!diff) return;
    uint32_t *w = reinterpret_cast<uint32_t *>(v.t);
    if (BPE == 1) atomicXor(w + (i >> 2), diff << (8 * (i & 3u)));
    else atomicXor(w + (i >> 1), (((diff & 0xFFu) << 8) | (diff >> 8)) << (16 * (i & 1u)));
}
// slot i's element becomes e, its occupied bit apart; each slot is set once
template <int BPE>
__device__ __forceinline__ void set_slot(const SlotTable<BPE> &v, uint32_t i, uint32_t e)
{
    xor_slot(v, i, (v.get(i) ^ e) & ~4u);
}
// Slots that one thread rewrites at the table's end, beside warps that change
// neighbouring slots with xor_slot: the same word atomics wherever the word is
// whole, single slots in the table's ragged last word, which xor_slot never
// touches.
template <int BPE>
struct EndSlots {
    const SlotTable<BPE> &v;
    __device__ __forceinline__ uint32_t get(uint32_t i) const
    {
        if (BPE == 1) return __ldcg(v.t + i);
        const uint32_t x = __ldcg(reinterpret_cast<const uint16_t *>(v.t) + i);
        return ((x & 0xFFu) << 8) | (x >> 8);
    }
    __device__ __forceinline__ void put(uint32_t i, uint32_t e) const
    {
        if ((i | (4 / BPE - 1)) < v.nslots) xor_slot(v, i, get(i) ^ e);
        else v.put(i, e);
    }
};
constexpr int LIST_THREADS = 64;

// ------------------------------------------------------------------ delete
// claim: two bits per slot, bit 0 "delete the element here", bit 1 "a thread
// has this unit" (at the unit's first slot).  lead[i]: the unit key i leads
// and what it claimed there: slot (UPD_NONE: none), slot - unit << 16 |
// unit end - slot, quotient, runs pending behind the slot.
template <int BPE>
__global__ void __launch_bounds__(UPD_THREADS) k_del_locate(const uint32_t *__restrict__ keys, uint32_t n,
                                                           SlotTable<BPE> v, uint32_t q, uint32_t r,
                                                           uint32_t *__restrict__ claim, uint4 *__restrict__ lead,
                                                           uint32_t *far)
{
    const uint32_t i = blockIdx.x * UPD_THREADS + threadIdx.x;
    if (i >= n) return;
    const uint32_t fp = aphash32(__ldg(keys + i)) & ((1u << (q + r)) - 1u);
    const uint32_t fq = fp >> r, fr = fp & ((1u << r) - 1u);
    Walk<BPE> k(v, fq);
    k.s.planes();
    uint4 mine = make_uint4(UPD_NONE, 0u, 0u, 0u);
    if ((k.s.occ >> (fq & 31u)) & 1u) {
        const uint32_t hocc = k.s.occ, hsi = k.si;
        const RunPlace p = find_run(k, fq);
        if (p.far) *far = 1;
        for (uint32_t s = p.pos; s < v.nslots && !p.far;) {
            const uint32_t e = k.elem(s);
            if (s > p.pos && !(e & 2u)) break;  // end of the run
            const uint32_t rem = e >> 3;
            if (rem > fr) break;
            if (rem < fr) {
                s++;
                continue;
            }
            // one copy per occurrence: the first copy nobody claimed.  Most
            // units are claimed once: the two claims and the unit's end are
            // asked for together.
            const uint32_t bit = 1u << (2 * (s & 15u));
            const uint32_t was = atomicOr(claim + (s >> 4), bit);
            if (!(was & bit)) {
                const uint32_t ub = 2u << (2 * (p.unit & 15u));
                if (!(atomicOr(claim + (p.unit >> 4), ub) & ub)) {
                    // quotients occupied in (fq, s]: fq's sector to the walk's
                    uint32_t D = 0;
                    for (uint32_t si = hsi; si <= (s >> 5); si++) {
                        uint32_t occ = si == k.si ? k.s.occ : hocc;
                        if (si != k.si && si != hsi) {
                            Sector<BPE> m;
                            m.load(v, si);
                            m.planes();
                            occ = m.occ;
                        }
                        if (si == hsi) occ &= ~low32((fq & 31u) + 1);
                        if (si == (s >> 5)) occ &= low32((s & 31u) + 1);
                        D += (uint32_t)__popc(occ);
                    }
                    const uint32_t end = k.first_clear(s + 1, [](const Sector<BPE> &x) { return x.sh; });
                    if (end == UPD_NONE || end - p.unit > v.far) *far = 1;
                    mine = make_uint4(s, ((s - p.unit) << 16) | (end - s), fq, D);
                }
                break;
            }
            // claimed: on to the next unclaimed slot of the claim word, unless
            // the run ends before it.  (A claim at a time, m deletes of one
            // fingerprint made m * m / 2 atomics: 208 ms for 30,000 copies.)
            const uint32_t open = ~was & 0x55555555u & (~0u << (2 * (s & 15u)));
            const uint32_t to = open ? (s & ~15u) + (((uint32_t)__ffs(open) - 1u) >> 1) : (s | 15u) + 1;
            if (k.s.rs & low32(min(to - (s & ~31u) + 1, 32u)) & ~low32((s & 31u) + 1)) break;
            if (to - p.pos > v.far || *reinterpret_cast<volatile uint32_t *>(far)) {
                *far = 1;
                break;
            }
            s = to;
        }
    }
    lead[i] = mine;
}

// Rewrites unit u without its claimed elements, slot by slot: every kept
// element goes to max(its quotient, the slot after the one before it).
template <typename Slots, typename Claimed>
__device__ __forceinline__ void del_unit(const Slots &v, Claimed &&claimed, uint32_t u, uint32_t end)
{
    uint32_t quot = u;  // quotient of the current run
    uint32_t c = u;     // first free slot
    uint32_t kept = 0;  // elements kept of the current run
    for (uint32_t t = u; t < end; t++) {
        const uint32_t e = v.get(t);
        if (t > u && !(e & 2u)) {  // a new run
            if (!kept) v.put(quot, v.get(quot) & ~4u);
            do quot++;
            while (quot < t && !(v.get(quot) & 4u));
            kept = 0;
        }
        if (claimed(t)) continue;
        for (; c < quot; c++) v.put(c, 0u);
        v.put(c, (e & ~7u) | (kept ? 2u : 0u) | (c != quot ? 1u : 0u) | (v.get(c) & 4u));
        c++;
        kept++;
    }
    if (!kept) v.put(quot, v.get(quot) & ~4u);
    for (; c < end; c++) v.put(c, 0u);
}

// A warp's lanes with `want` append x to the list.
template <typename T>
__device__ __forceinline__ void append(T *list, uint32_t *count, bool want, const T &x)
{
    const unsigned m = __ballot_sync(__activemask(), want);
    if (!want) return;
    const unsigned lane = threadIdx.x & 31, first = (unsigned)__ffs(m) - 1u;
    uint32_t base = 0;
    if (lane == first) base = atomicAdd(count, (uint32_t)__popc(m));
    base = __shfl_sync(m, base, (int)first);
    list[base + (uint32_t)__popc(m & ((1u << lane) - 1u))] = x;
}

// One thread per led unit with one claimed element: the rest moves by one
// slot, a word at a time.  Units with more claims, a fifth of the keys at
// 2^20 deletes from a 2^26 table, are listed for k_del_units: they walk slot
// by slot, and in this kernel every warp would wait for a few of them.
template <int BPE>
__global__ void __launch_bounds__(UPD_THREADS) k_del_apply(uint32_t n, SlotTable<BPE> v,
                                                          const uint32_t *__restrict__ claim,
                                                          const uint4 *__restrict__ lead, uint2 *__restrict__ units,
                                                          uint32_t *__restrict__ n_units,
                                                          const uint32_t *__restrict__ far)
{
    const uint32_t i = blockIdx.x * UPD_THREADS + threadIdx.x;
    if (*far) return;
    const uint4 l = i < n ? lead[i] : make_uint4(UPD_NONE, 0u, 0u, 0u);
    const uint32_t s = l.x, u = s - (l.y >> 16), end = s + (l.y & 0xFFFFu);
    bool single = false;
    if (BPE == 1 && s != UPD_NONE && (end | 31u) < v.nslots) {
        // another of the unit's elements claimed?
        uint32_t all = 0;
        for (uint32_t c = u >> 4; c <= ((end - 1) >> 4); c++) {
            const int a = max((int)u - (int)(16 * c), 0), b = min((int)end - (int)(16 * c), 16);
            const uint32_t in = (b >= 16 ? ~0u : (1u << (2 * b)) - 1u) & ~((1u << (2 * a)) - 1u);
            all += (uint32_t)__popc(claim[c] & 0x55555555u & in);
        }
        single = all == 1;
    }
    __syncwarp();
    append(units, n_units, s != UPD_NONE && !single, make_uint2(u, end));
    if constexpr (BPE == 1)
        if (single) shift_left(v, s, end, l.z, l.w);
}

// The same by a warp, 32 slots at a time, a lane per slot.  The j-th run
// start of the 32 belongs to the j-th occupied quotient after the current
// run's; an element's slot is a running maximum over the kept ones of
// (quotient - number of kept ones before), plus that number.
template <int BPE>
__device__ __forceinline__ void del_unit_warp(const SlotTable<BPE> &v, const uint32_t *__restrict__ claim, uint32_t u,
                                              uint32_t end)
{
    const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    uint32_t quot = u, c = u;  // the current run's quotient, the first free slot
    bool kept = false;         // an element of the current run was kept
    for (uint32_t t0 = u; t0 < end;) {
        const uint32_t slot = t0 + lane;
        bool in = slot < end;
        const uint32_t e = in ? v.get(slot) : 0u;
        const bool cl = in && ((claim[slot >> 4] >> (2 * (slot & 15u))) & 1u);
        uint32_t rs = __ballot_sync(~0u, in && !(e & 2u) && slot > u);
        // the next occupied quotients: 64 from qb on
        uint32_t qb = quot + 1, m0, m1;
        for (;; qb += 64) {
            const uint32_t a = qb + lane, b = qb + 32 + lane;
            m0 = __ballot_sync(~0u, a < end && (v.get(a) & 4u));
            m1 = __ballot_sync(~0u, b < end && (v.get(b) & 4u));
            if (m0 | m1 | !rs || qb + 64 >= end) break;
        }
        const uint32_t n0 = (uint32_t)__popc(m0), na = n0 + (uint32_t)__popc(m1);
        uint32_t adv = 32;
        if ((uint32_t)__popc(rs) > na) {  // as far as the quotients at hand go
            adv = max(nth_bit(rs, (int)na), 1u);
            in = in && lane < adv;
            rs &= low32(adv);
        }
        const uint32_t j = (uint32_t)__popc(rs & lt);
        uint32_t mine = 0;  // a run start's quotient
        if ((rs >> lane) & 1u)
            mine = j < n0 ? qb + nth_bit(m0, (int)j) : j < na ? qb + 32 + nth_bit(m1, (int)(j - n0)) : slot;
        const uint32_t upto = rs & (lt | (1u << lane));
        const bool carried = !upto;  // still in the run the 32 slots began in
        const uint32_t h = carried ? 0u : 31u - (uint32_t)__clz(upto);
        const uint32_t from_h = __shfl_sync(~0u, mine, (int)h);
        const uint32_t K = carried ? quot : from_h;
        const bool live = in && !cl;
        const uint32_t sv = __ballot_sync(~0u, live), rank = (uint32_t)__popc(sv & lt);
        int M = live ? (int)K - (int)rank : -0x40000000;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(~0u, M, o);
            if ((int)lane >= o) M = max(M, y);
        }
        const uint32_t pos = (uint32_t)(max(M, (int)c) + (int)rank);
        const uint32_t before = sv & lt & ~low32(h);
        const uint32_t prev = __shfl_sync(~0u, pos, (sv & lt) ? 31 - __clz(sv & lt) : 0);
        if (live) {
            for (uint32_t x = rank ? prev + 1 : c; x < pos; x++) set_slot(v, x, 0u);  // slots left empty
            set_slot(v, pos, (e & ~7u) | ((before || (carried && kept)) ? 2u : 0u) | (pos != K ? 1u : 0u));
        }
        // runs that ended here without a kept element: their quotients are free
        if ((rs >> lane) & 1u) {
            const uint32_t later = rs & ~(lt | (1u << lane));
            if (later && !(sv & low32((uint32_t)__ffs(later) - 1u) & ~lt)) xor_slot(v, mine, 4u);
        }
        if (rs && lane == 0 && !kept && !(sv & low32((uint32_t)__ffs(rs) - 1u))) xor_slot(v, quot, 4u);
        const uint32_t lastpos = __shfl_sync(~0u, pos, sv ? 31 - __clz(sv) : 0);
        if (sv) c = lastpos + 1;
        if (rs) {
            const uint32_t l = 31u - (uint32_t)__clz(rs);
            quot = __shfl_sync(~0u, mine, (int)l);
            kept = (sv & ~low32(l)) != 0;
        } else {
            kept = kept || sv != 0;
        }
        t0 += adv;
    }
    if (lane == 0 && !kept) xor_slot(v, quot, 4u);
    for (uint32_t x = c + lane; x < end; x += 32) set_slot(v, x, 0u);
}

// The listed units, a warp each (those in the table's last word, which is not
// whole, by one lane).
template <int BPE>
__global__ void __launch_bounds__(LIST_THREADS) k_del_units(SlotTable<BPE> v, const uint32_t *__restrict__ claim,
                                                           const uint2 *__restrict__ units,
                                                           const uint32_t *__restrict__ n_units)
{
    const uint32_t n = *n_units;
    for (uint32_t i = (blockIdx.x * LIST_THREADS + threadIdx.x) >> 5; i < n; i += gridDim.x * (LIST_THREADS / 32)) {
        const uint2 un = units[i];
        if ((un.y | 3u) < v.nslots)
            del_unit_warp(v, claim, un.x, un.y);
        else if ((threadIdx.x & 31) == 0)
            del_unit(EndSlots<BPE>{v}, [&](uint32_t t) { return (claim[t >> 4] >> (2 * (t & 15u))) & 1u; }, un.x, un.y);
        __syncwarp();
    }
}

// ------------------------------------------------------------------ insert
// The batch's new fingerprints: bucket b (quotient range fp >> shift) holds
// cnt[b] of them from base[b], sorted by k_ins_sort, as entries
//   x  fingerprint
//   y  slot the key goes in front of; INS_HEAD: in front of its run's first
//      element, or first of a new run
//   z  first empty slot at or after its quotient; INS_NEWQ: its quotient has
//      no run yet; INS_COVERED (first key of a gap): an earlier gap's inserts
//      reach this one's cluster
constexpr uint32_t INS_HEAD = 1u << 31, INS_COVERED = 1u << 31, INS_NEWQ = 1u << 30;
constexpr uint32_t INS_GAP = INS_NEWQ - 1;

struct InsBatch {
    uint32_t nb, shift, stride, hmask;
    uint32_t *cnt, *base;     // per bucket
    uint32_t *n_over, *pool;  // keys past their bucket's stride; pool space handed out
    uint32_t *n_group;        // groups of several keys
    uint4 *key;               // nb * stride entries, then the pool of n
    uint4 *over;              // n: the overflow list, then the groups of several keys (last key, last gap)
    uint32_t *seen;           // hash set of hmask + 1 entries, all ones
};

template <int BPE>
__global__ void __launch_bounds__(UPD_THREADS) k_ins_stage(const uint32_t *__restrict__ keys, uint32_t n,
                                                          SlotTable<BPE> v, uint32_t q, uint32_t r, InsBatch b,
                                                          uint32_t *far)
{
    const uint32_t i = blockIdx.x * UPD_THREADS + threadIdx.x;
    if (i >= n) return;
    const uint32_t fp = aphash32(__ldg(keys + i)) & ((1u << (q + r)) - 1u);
    const uint32_t fq = fp >> r, fr = fp & ((1u << r) - 1u);
    // repeated in the batch: only the thread whose entry this is goes on
    uint32_t h = (fp * 0x9E3779B1u) >> 7;
    uint32_t cur = *reinterpret_cast<volatile uint32_t *>(b.seen + (h & b.hmask));
    Walk<BPE> w(v, fq);  // in flight beside the set's entry
    for (uint32_t tries = 0; tries <= b.hmask; tries++) {
        uint32_t *slot = b.seen + (h & b.hmask);
        if (tries) cur = *reinterpret_cast<volatile uint32_t *>(slot);
        if (cur == UPD_NONE) cur = atomicCAS(slot, UPD_NONE, fp);
        if (cur == UPD_NONE) break;
        if (cur == fp) return;
        h++;
    }
    w.s.planes();
    const RunPlace p = find_run(w, fq);
    uint32_t ip = p.pos, head = INS_HEAD;
    if (p.occ && !p.far) {
        for (; ip < v.nslots && ip - p.pos <= v.far; ip++) {
            const uint32_t e = w.elem(ip);
            if (ip > p.pos && !(e & 2u)) break;  // end of the run
            const uint32_t rem = e >> 3;
            if (rem == fr) return;  // stored already
            if (rem > fr) break;
        }
        if (ip != p.pos) head = 0;
    }
    const uint32_t gap = p.far || ip - p.pos > v.far ? UPD_NONE : ip >= v.nslots ? v.nslots : w.next_empty(ip);
    if (gap == UPD_NONE) *far = 1;
    const uint4 entry = make_uint4(fp, ip | head, (gap & INS_GAP) | (p.occ ? 0u : INS_NEWQ), 0u);
    const uint32_t bk = fp >> b.shift, k = atomicAdd(b.cnt + bk, 1u);
    if (k < b.stride) b.key[(size_t)bk * b.stride + k] = entry;
    else b.over[atomicAdd(b.n_over, 1u)] = entry;
}

// Ascending sort of m (fingerprint, index) words by the CTA (all comparators
// ascending, so the missing tail of the last power of two acts as the
// largest values).
template <int THREADS, typename T, typename Key>
__device__ __forceinline__ void cta_sort(T *a, uint32_t m, Key &&key)
{
    uint32_t p2 = 1;
    while (p2 < m) p2 <<= 1;
    for (uint32_t k = 2; k <= p2; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            const bool flip = j == (k >> 1);
            for (uint32_t i = threadIdx.x; i < p2 / 2; i += THREADS) {
                const uint32_t lo = 2 * i - (i & (j - 1)), hi = flip ? (lo ^ (k - 1)) : lo + j;
                if (hi < m) {
                    const T x = a[lo], y = a[hi];
                    if (key(x) > key(y)) {
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
constexpr uint32_t INS_SMEM_KEYS = 512;

// Sorts each bucket's entries by fingerprint: through (fingerprint, index)
// pairs in shared memory, or, past INS_SMEM_KEYS entries (keys crowded into
// few quotients), the entries themselves in global memory.
static __global__ void __launch_bounds__(INS_THREADS) k_ins_sort(InsBatch b, const uint32_t *__restrict__ far)
{
    __shared__ unsigned long long s_key[INS_SMEM_KEYS];
    __shared__ uint4 s_ent[INS_SMEM_KEYS];
    __shared__ uint32_t s_n, s_base;
    if (*far) return;
    const uint32_t bk = blockIdx.x, cnt = b.cnt[bk], tid = threadIdx.x;
    if (cnt == 0) return;
    uint32_t base = bk * b.stride;
    uint4 *ent = b.key + base;
    if (cnt > b.stride) {  // the keys past the region are in the overflow list: gather all in the pool
        if (tid == 0) {
            s_base = b.nb * b.stride + atomicAdd(b.pool, cnt);
            s_n = b.stride;
        }
        __syncthreads();
        base = s_base;
        for (uint32_t i = tid; i < b.stride; i += INS_THREADS) b.key[base + i] = ent[i];
        ent = b.key + base;
        const uint32_t no = *b.n_over;
        for (uint32_t i = tid; i < no; i += INS_THREADS) {
            const uint4 e = b.over[i];
            if ((e.x >> b.shift) == bk) ent[atomicAdd(&s_n, 1u)] = e;
        }
        __syncthreads();
    }
    if (tid == 0) b.base[bk] = base;
    if (cnt <= INS_SMEM_KEYS) {
        for (uint32_t i = tid; i < cnt; i += INS_THREADS) {
            const uint4 e = ent[i];
            s_ent[i] = e;
            s_key[i] = ((unsigned long long)e.x << 32) | i;
        }
        __syncthreads();
        cta_sort<INS_THREADS>(s_key, cnt, [](unsigned long long x) { return x; });
        for (uint32_t i = tid; i < cnt; i += INS_THREADS) ent[i] = s_ent[(uint32_t)s_key[i]];
    } else {
        cta_sort<INS_THREADS>(ent, cnt, [](const uint4 &x) { return x.x; });
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
    const uint32_t g = b.key[ins_at(b, k)].z & INS_GAP;
    InsPos p = k;
    return !ins_prev(b, p) || (b.key[ins_at(b, p)].z & INS_GAP) != g;
}
// From the first key k of gap g: takes the keys of one gap after the other
// until their empty slots have taken every shift.  Returns the last gap
// (nslots: the table is full), the last key taken in `last`; mark(key) for
// the first key of every gap after the first.
template <int BPE, typename Mark>
__device__ __forceinline__ uint32_t ins_walk(const InsBatch &b, const SlotTable<BPE> &v, InsPos k, InsPos &last,
                                             Mark &&mark, uint32_t *taken = nullptr)
{
    uint32_t pending = 0, g = b.key[ins_at(b, k)].z & INS_GAP;
    const uint32_t g0 = g;
    for (;;) {
        if (g != g0 && ins_valid(b, k) && (b.key[ins_at(b, k)].z & INS_GAP) == g && !mark(ins_at(b, k))) return g;
        while (ins_valid(b, k) && (b.key[ins_at(b, k)].z & INS_GAP) == g) {
            pending++;
            if (taken) ++*taken;
            last = k;
            k = ins_next(b, k);
        }
        if (g >= v.nslots || --pending == 0) return g;
        if (g + 1 >= v.nslots) return v.nslots;
        Walk<BPE> w(v, g + 1);
        w.s.planes();
        g = w.next_empty(g + 1);
        if (g - g0 > v.far) return g == v.nslots ? g : UPD_NONE;
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
        const volatile uint32_t *own = &b.key[ins_at(b, k)].z;
        if (ins_walk<BPE>(b, v, k, last, [&](uint32_t at) {
                atomicOr(&b.key[at].z, INS_COVERED);
                return !(*own & INS_COVERED);
            }) == UPD_NONE)
            *far = 1;
    }
}

// Puts in the keys up to `last` of a group whose shifts end in empty slot g,
// from right to left, slot by slot: d = slots an element here moves.
template <typename Slots>
__device__ __forceinline__ void ins_group(const Slots &v, uint32_t r, const InsBatch &b, InsPos k, uint32_t g)
{
    uint4 ent = b.key[ins_at(b, k)];
    uint32_t d = 0;
    for (uint32_t s = g;; s--) {
        const uint32_t e = v.get(s);
        const bool here = (ent.y & ~INS_HEAD) == s;
        if (!(e & 7u)) {
            d++;  // an empty slot takes one shift
        } else {
            // the old head of a run continues it when a new key goes in front
            const uint32_t cont = (here && (ent.y & INS_HEAD) && !(ent.z & INS_NEWQ)) ? 2u : 0u;
            v.put(s + d, (e & ~4u) | 1u | cont | (v.get(s + d) & 4u));
        }
        while ((ent.y & ~INS_HEAD) == s) {
            const uint32_t fp = ent.x, fq = fp >> r, pos = s + d - 1;
            const bool newq = (ent.z & INS_NEWQ) != 0, head = (ent.y & INS_HEAD) != 0;
            d--;
            bool behind = false;  // a smaller new key of the same quotient
            const bool more = ins_prev(b, k);
            if (more) {
                ent = b.key[ins_at(b, k)];
                behind = (ent.x >> r) == fq;
            }
            v.put(pos, ((fp & ((1u << r) - 1u)) << 3) | ((head && !behind) ? 0u : 2u) | (pos != fq ? 1u : 0u) |
                           (v.get(pos) & 4u));
            if (newq && !behind) v.put(fq, v.get(fq) | 4u);
            if (!d || !more) break;
        }
        if (!d) break;
    }
}

// One thread per group of one key: the elements behind it move by one slot, a
// word at a time.  Groups of more keys are listed for k_ins_lists.
template <int BPE>
__global__ void __launch_bounds__(INS_THREADS) k_ins_apply(SlotTable<BPE> v, uint32_t r, InsBatch b, uint32_t *err,
                                                          const uint32_t *__restrict__ far)
{
    if (*far) return;
    const uint32_t bk = blockIdx.x, cnt = b.cnt[bk];
    for (uint32_t i0 = 0; i0 < cnt; i0 += INS_THREADS) {
        const uint32_t i = i0 + threadIdx.x;
        const InsPos k{bk, i};
        InsPos last = k;
        uint4 ent = make_uint4(0u, 0u, INS_COVERED, 0u);
        if (i < cnt) ent = b.key[ins_at(b, k)];
        uint32_t g = UPD_NONE, taken = 0;
        if (!(ent.z & INS_COVERED) && ins_first(b, k)) {
            g = ins_walk<BPE>(b, v, k, last, [](uint32_t) { return true; }, &taken);
            if (g >= v.nslots) {
                atomicOr(err, DEV_ERR_FULL);
                g = UPD_NONE;
            }
        }
        const bool single = BPE == 1 && g != UPD_NONE && (g | 31u) < v.nslots && last.bk == bk && last.i == i;
        __syncwarp();
        append(b.over, b.n_group, g != UPD_NONE && !single, make_uint4(last.bk, last.i, g, taken));
        if constexpr (BPE == 1) {
            if (single) {
                const uint32_t fq = ent.x >> r, ip = ent.y & ~INS_HEAD;
                const bool head = (ent.y & INS_HEAD) != 0, newq = (ent.z & INS_NEWQ) != 0;
                shift_right(v, ip, g, ((ent.x & ((1u << r) - 1u)) << 3) | (head ? 0u : 2u) | (ip != fq ? 1u : 0u),
                            head && !newq);
                if (newq) xorw(v, fq >> 3, 4ull << (8 * (fq & 7u)));  // (one word size per launch)
            }
        }
    }
}

// ins_group by a warp for a group of nk keys: 32 slots at a time from the
// right, a lane per slot.  The shift at a slot is the shift behind the 32
// plus the empty slots less the keys between.
struct InsCounts {
    uint32_t keys[32], cont[32], above[32];
    int shift[32];
};
template <int BPE>
__device__ __forceinline__ void ins_group_warp(const SlotTable<BPE> &v, uint32_t r, const InsBatch &b, InsPos k,
                                               uint32_t g, uint32_t nk, InsCounts &sc)
{
    const uint32_t lane = threadIdx.x & 31;
    int d = 0;
    // f(entry, index from the top, smaller key of the same quotient?) for the
    // group's keys going in front of slots of sector si, from the top; returns
    // their number and leaves k behind them
    auto keys_of = [&](uint32_t si, InsPos &at, uint32_t left, auto &&f) -> uint32_t {
        uint32_t total = 0;
        while (total < left) {
            const uint4 *top = b.key + ins_at(b, at);
            const bool have = lane <= at.i && total + lane < left;
            const uint4 e = have ? *(top - lane) : make_uint4(0u, 0u, 0u, 0u);
            const bool mine = have && ((e.y & ~INS_HEAD) >> 5) == si;
            const uint32_t m = __ballot_sync(~0u, mine), nv = (uint32_t)__popc(m);
            if (mine) f(e, total + lane, at.i > lane && ((top - lane - 1)->x >> r) == (e.x >> r));
            total += nv;
            if (nv == 0) break;
            if (nv <= at.i) {
                at.i -= nv;
            } else {  // on to the bucket before (another bucket, another quotient)
                at.i = 0;
                if (!ins_prev(b, at)) break;
            }
        }
        return total;
    };
    for (uint32_t si = g >> 5;; si--) {
        const uint32_t s = 32 * si + lane;
        const bool in = s <= g;
        const uint32_t e = in ? v.get(s) : 1u;
        sc.keys[lane] = sc.cont[lane] = 0;
        __syncwarp();
        InsPos at = k;
        const uint32_t n = keys_of(si, at, nk, [&](const uint4 &x, uint32_t, bool) {
            const uint32_t p = x.y & 31u;
            atomicAdd(&sc.keys[p], 1u);
            // the old head of a run continues it when a new key goes in front
            if ((x.y & INS_HEAD) && !(x.z & INS_NEWQ)) sc.cont[p] = 2u;
        });
        __syncwarp();
        const bool gap = in && !(e & 7u);
        const uint32_t nkeys = sc.keys[lane];
        int suf = (gap ? 1 : 0) - (int)nkeys;
        uint32_t kab = nkeys;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_down_sync(~0u, suf, o);
            const uint32_t z = __shfl_down_sync(~0u, kab, o);
            if (lane + o < 32) {
                suf += y;
                kab += z;
            }
        }
        const int ds = d + suf - ((gap ? 1 : 0) - (int)nkeys);
        sc.shift[lane] = ds + (gap ? 1 : 0);
        sc.above[lane] = kab - nkeys;
        const int dn = d + __shfl_sync(~0u, suf, 0);
        // (slots in front of the group's first key stay)
        if (in && !gap && nk > kab - nkeys) set_slot(v, s + (uint32_t)ds, (e & ~4u) | 1u | sc.cont[lane]);
        __syncwarp();
        at = k;
        keys_of(si, at, nk, [&](const uint4 &x, uint32_t idx, bool behind) {
            const uint32_t p = x.y & 31u, fq = x.x >> r, head = x.y & INS_HEAD;
            const uint32_t pos = 32 * si + p + (uint32_t)sc.shift[p] - 1u - (idx - sc.above[p]);
            set_slot(v, pos, ((x.x & ((1u << r) - 1u)) << 3) | ((head && !behind) ? 0u : 2u) | (pos != fq ? 1u : 0u));
            if ((x.z & INS_NEWQ) && !behind) xor_slot(v, fq, 4u);
        });
        k = at;
        nk -= n;
        d = dn;
        __syncwarp();
        if (nk == 0 || si == 0) break;
    }
}

template <int BPE>
__global__ void __launch_bounds__(LIST_THREADS) k_ins_lists(SlotTable<BPE> v, uint32_t r, InsBatch b)
{
    __shared__ InsCounts sc[LIST_THREADS / 32];
    const uint32_t n = *b.n_group;
    for (uint32_t i = (blockIdx.x * LIST_THREADS + threadIdx.x) >> 5; i < n; i += gridDim.x * (LIST_THREADS / 32)) {
        const uint4 e = b.over[i];  // last key, last gap, keys
        if ((e.z | 3u) < v.nslots)
            ins_group_warp(v, r, b, InsPos{e.x, e.y}, e.z, e.w, sc[threadIdx.x >> 5]);
        else if ((threadIdx.x & 31) == 0)
            ins_group(EndSlots<BPE>{v}, r, b, InsPos{e.x, e.y}, e.z);
        __syncwarp();
    }
}

}  // namespace gqf

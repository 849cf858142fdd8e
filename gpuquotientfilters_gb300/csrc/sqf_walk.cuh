// Walks over the table, 32 slots per memory round trip: where a quotient's
// run is, the next empty slot, the end of a shifted stretch.  Shared by the
// updates and the lookups on two-byte slots.
#pragma once

#include "qf_device.cuh"

namespace gqf {

constexpr uint32_t WALK_NONE = 0xFFFFFFFFu;
// A longer stretch (a nearly full table) is not walked: SlotTable::far slots
// for an update, FAR_SLOTS at most.  An update that meets one sets *far:
// nothing has been changed yet, the apply kernels do nothing, and the table is
// updated as a whole.  A lookup goes on slot by slot.
constexpr uint32_t FAR_SLOTS = 5120;

// Slots of a table: element i = rem << 3 | occupied << 2 |
// continuation << 1 | shifted.
template <int BPE>
struct SlotTable {
    uint8_t *t;
    uint32_t nslots, far = FAR_SLOTS;
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
};

// 32 consecutive slots: their bit planes (bit i = slot 32 * index + i) and,
// for one-byte slots, their bytes.  A walk takes a sector per memory round
// trip; slot by slot or word by word, the longest walk of a warp's 32 took
// most of the time.
template <int BPE>
struct Sector {
    uint64_t w[4];
    uint32_t occ, rs, sh, ne;
    __device__ __forceinline__ void load(const SlotTable<BPE> &v, uint32_t index)
    {
        const uint32_t s0 = 32 * index;
        if constexpr (BPE == 1) {
            if (s0 + 32 <= v.nslots) {
                const ulonglong2 a = __ldcg(reinterpret_cast<const ulonglong2 *>(v.t + s0));
                const ulonglong2 b = __ldcg(reinterpret_cast<const ulonglong2 *>(v.t + s0) + 1);
                w[0] = a.x;
                w[1] = a.y;
                w[2] = b.x;
                w[3] = b.y;
            } else {
                for (int j = 0; j < 4; j++) {
                    w[j] = 0;
                    for (uint32_t k = 0; k < 8; k++) {
                        const uint32_t i = s0 + 8 * j + k;
                        if (i < v.nslots) w[j] |= (uint64_t)v.t[i] << (8 * k);
                    }
                }
            }
        } else if (s0 + 32 <= v.nslots) {
            // a slot's flags are in the second (low) byte of its two
            auto nib = [](uint64_t x) -> uint32_t {
                return (uint32_t)(((x & 0x0001000100010001ull) * 0x0001000200040008ull) >> 48) & 15u;
            };
            uint32_t cont = 0;
            occ = sh = 0;
            const ulonglong2 *p = reinterpret_cast<const ulonglong2 *>(v.t + 2 * (size_t)s0);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const ulonglong2 a = __ldcg(p + j);
                sh |= (nib(a.x >> 8) | (nib(a.y >> 8) << 4)) << (8 * j);
                cont |= (nib(a.x >> 9) | (nib(a.y >> 9) << 4)) << (8 * j);
                occ |= (nib(a.x >> 10) | (nib(a.y >> 10) << 4)) << (8 * j);
            }
            ne = occ | cont | sh;
            rs = (occ | sh) & ~cont;
        } else {
            occ = rs = sh = ne = 0;
            for (uint32_t k = 0; k < 32; k++) {
                const uint32_t e = s0 + k < v.nslots ? v.get(s0 + k) : 0u;
                occ |= ((e >> 2) & 1u) << k;
                sh |= (e & 1u) << k;
                ne |= ((e & 7u) ? 1u : 0u) << k;
                rs |= (((e & 7u) && !(e & 2u)) ? 1u : 0u) << k;
            }
        }
    }
    // the planes of one-byte slots (apart from the load, so that other loads
    // can be in flight between)
    __device__ __forceinline__ void planes()
    {
        if constexpr (BPE == 1) {
            auto nib = [](uint32_t x) -> uint32_t { return ((x & 0x01010101u) * 0x01020408u) >> 24; };
            uint32_t cont = 0;
            occ = sh = 0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t lo = (uint32_t)w[j], hi = (uint32_t)(w[j] >> 32);
                sh |= (nib(lo) | (nib(hi) << 4)) << (8 * j);
                cont |= (nib(lo >> 1) | (nib(hi >> 1) << 4)) << (8 * j);
                occ |= (nib(lo >> 2) | (nib(hi >> 2) << 4)) << (8 * j);
            }
            ne = occ | cont | sh;
            rs = (occ | sh) & ~cont;
        }
    }
    __device__ __forceinline__ uint32_t elem(const SlotTable<BPE> &v, uint32_t i) const  // slot i of this sector
    {
        if constexpr (BPE == 1) {
            const uint32_t j = (i >> 3) & 3u;
            const uint64_t x = j & 2u ? (j & 1u ? w[3] : w[2]) : (j & 1u ? w[1] : w[0]);
            return (uint32_t)(x >> (8 * (i & 7u))) & 0xFFu;
        } else {
            return i < v.nslots ? v.get(i) : 0u;
        }
    }
};
__device__ __forceinline__ uint32_t low32(uint32_t n) { return n >= 32 ? ~0u : (1u << n) - 1u; }

// A position in the table with its sector.
template <int BPE>
struct Walk {
    const SlotTable<BPE> &v;
    Sector<BPE> s;
    uint32_t si;
    __device__ __forceinline__ Walk(const SlotTable<BPE> &t, uint32_t slot) : v(t), si(slot >> 5) { s.load(v, si); }
    __device__ __forceinline__ void to(uint32_t slot)
    {
        if ((slot >> 5) != si) {
            si = slot >> 5;
            s.load(v, si);
            s.planes();
        }
    }
    __device__ __forceinline__ uint32_t elem(uint32_t slot)
    {
        to(slot);
        return s.elem(v, slot);
    }
    // first slot at or after `slot` for which the plane pick(sector) is clear
    // (the table's end reads as clear; WALK_NONE: further than v.far)
    template <typename Pick>
    __device__ __forceinline__ uint32_t first_clear(uint32_t slot, Pick &&pick)
    {
        const uint32_t from = slot;
        for (;;) {
            to(slot);
            const uint32_t m = ~pick(s) & ~low32(slot & 31u);
            if (m) return min(32 * si + (uint32_t)__ffs(m) - 1u, v.nslots);
            slot = 32 * si + 32;
            if (slot >= v.nslots) return v.nslots;
            if (slot - from > v.far) return WALK_NONE;
        }
    }
    // first empty slot at or after `slot` (nslots: none)
    __device__ __forceinline__ uint32_t next_empty(uint32_t slot)
    {
        return first_clear(slot, [](const Sector<BPE> &x) { return x.ne; });
    }
};

// Where quotient fq's run is or would go, from the unchanged table; the walk
// starts in fq's sector (planes taken) and ends in pos's.
//   unit: the last unshifted slot at or below fq (the start of fq's unit when
//         fq is occupied);
//   occ:  fq has a run;
//   pos:  occ: the run's first slot; otherwise the slot a first element of fq
//         goes in front of (the next run's start or the first empty slot);
//   far:  the walk went past k.v.far, pos is not known.
struct RunPlace {
    uint32_t unit, pos;
    bool occ, far;
};
template <int BPE>
__device__ __forceinline__ RunPlace find_run(Walk<BPE> &k, uint32_t fq)
{
    RunPlace r;
    r.far = false;
    r.pos = k.v.nslots;
    const uint32_t at = fq & 31u;
    r.occ = (k.s.occ >> at) & 1u;
    // back to the last unshifted slot; D = runs of lower quotients starting
    // at or after fq
    int D = 0;
    {
        Sector<BPE> b = k.s;
        uint32_t bi = k.si, in = low32(at), st = ~b.sh & low32(at + 1);
        while (!st) {
            D += __popc(b.occ & in) - __popc(b.rs & in);
            if (bi == 0) break;
            if (k.si - bi > k.v.far / 32) {
                r.far = true;
                return r;
            }
            b.load(k.v, --bi);
            b.planes();
            in = ~0u;
            st = ~b.sh;
        }
        const uint32_t hb = st ? 31u - (uint32_t)__clz(st) : 0u;
        if (st) {
            in &= ~low32(hb);
            D += __popc(b.occ & in) - __popc(b.rs & in);
        }
        r.unit = 32 * bi + hb;
    }
    // forward to the (D+1)-th run start; without a run of fq, no further
    // than the first empty slot
    uint32_t from = ~low32(at);
    for (;;) {
        const uint32_t rs = k.s.rs & from, em = ~k.s.ne & from;
        const int c = __popc(rs);
        uint32_t p = 32;
        if (c > max(D, 0)) p = nth_bit(rs, max(D, 0));
        if (!r.occ && em) p = min(p, (uint32_t)__ffs(em) - 1u);
        if (p < 32) {
            r.pos = min(32 * k.si + p, k.v.nslots);
            return r;
        }
        D -= c;
        const uint32_t next = 32 * k.si + 32;
        if (next >= k.v.nslots) return r;
        if (next - fq > k.v.far) {
            r.far = true;
            return r;
        }
        k.to(next);
        from = ~0u;
    }
}

}  // namespace gqf

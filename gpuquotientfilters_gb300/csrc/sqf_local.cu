// Cluster-local inserts and deletes, with the general path behind them.
#include "sqf_fallback.cuh"
#include "sqf_host.cuh"
#include "sqf_update.cuh"

namespace gqf {

// ------------------------------------------------------ cluster-local updates
template <int BPE>
int local_update(const gqf_sqf *qf, const uint32_t *keys, uint32_t n, int op, cudaStream_t s, float *ms)
{
    const SqfGeom tg = geom_of(qf);
    const DeviceInfo &di = device_info(current_device());
    const bool ins = op == OP_INSERT;
    // insert buckets of about 128 keys, one CTA each
    InsBatch ib{};
    uint32_t lg = 0;
    while ((128ull << lg) < n && lg < std::min<uint32_t>(tg.q, 18)) lg++;
    ib.nb = 1u << lg;
    ib.shift = tg.q + tg.r - lg;
    const double avg = (double)n / ib.nb;
    ib.stride = (uint32_t)align_up((size_t)(avg + 10.0 * std::sqrt(avg) + 32.0), 32);
    uint32_t hsize = 1024;
    while (hsize < 2ull * n) hsize <<= 1;
    ib.hmask = hsize - 1;
    const size_t nkey = (size_t)ib.nb * ib.stride + n;
    // a table shorter than any walk's limit needs no fallback
    const bool fb = tg.nslots > FAR_SLOTS;
    static_assert((uint64_t)((1u << (FB_TB - 1)) * 1.1) <= FAR_SLOTS, "a fallback table spans whole buckets");
    const uint32_t fnb = fb ? 1u << (tg.q - FB_TB) : 1u;
    const uint32_t ntiles = (tg.nslots + EXTRACT_TILE - 1) / EXTRACT_TILE;
    FallbackArgs f{};
    uint32_t *far = nullptr, *claim = nullptr, *n_units = nullptr;
    uint2 *units = nullptr;
    uint4 *lead = nullptr;
    size_t zero_bytes = 0;
    // control words | delete claims (both zeroed) | then either the update's
    // arrays or, when the fallback runs, its own over them
    auto lay = [&](auto &c) {
        far = c.template take<uint32_t>(1);
        f.bar = c.template take<uint32_t>(4, 16);
        f.lay.ticket = c.template take<uint32_t>(1, 4);
        f.lay.fix_cnt = c.template take<uint32_t>(1, 4);
        ib.n_over = c.template take<uint32_t>(1, 4);
        ib.pool = c.template take<uint32_t>(1, 4);
        n_units = ib.n_group = c.template take<uint32_t>(1, 4);
        f.bcnt = c.template take<uint32_t>(fnb, 4);
        f.bfill = c.template take<uint32_t>(fnb, 4);
        f.lay.status = c.template take<unsigned long long>(fnb, 8);
        if (ins) ib.cnt = c.template take<uint32_t>(ib.nb, 4);
        else claim = c.template take<uint32_t>(2 * ((tg.nslots + 31) / 32), 16);
        zero_bytes = c.off;
        const size_t at = c.off;
        if (ins) {
            ib.seen = c.template take<uint32_t>(hsize);
            ib.base = c.template take<uint32_t>(ib.nb);
            ib.key = c.template take<uint4>(nkey);
            ib.over = c.template take<uint4>(n);
        } else {
            lead = c.template take<uint4>(n);
            units = c.template take<uint2>(n);
        }
        const size_t end = c.off;
        if (fb) {
            c.off = at;
            f.tiles = c.template take<Counts3>(ntiles + 1);
            f.Q = c.template take<uint32_t>(tg.nslots);
            f.E = c.template take<uint32_t>(tg.nslots);
            f.abase = c.template take<uint32_t>(fnb + 1);
            f.acnt = c.template take<uint32_t>(fnb);
            f.bbase = c.template take<uint32_t>(fnb + 1);
            f.bitems = c.template take<uint32_t>(n);
            // a fix-up for every quotient: on an overfull table the spill
            // passes whole buckets (the extraction is done with Q by then)
            f.lay.fix_cap = tg.nslots;
            f.lay.fix_list = f.Q;
            c.off = std::max(c.off, end);
        }
    };
    Sizer z;
    lay(z);
    Arena &ar = arena(current_device(), s);
    std::lock_guard<std::mutex> lk(ar.mu);
    void *base = arena_reserve(ar, z.off);
    if (!base) return GQF_ERR_NOMEM;
    Carver c(base);
    lay(c);
    int st = call_begin(ar, s, ms != nullptr);
    if (st) return st;
    if (n == 0) return call_end(ar, s, ms);
    GQF_CK(cudaMemsetAsync(base, 0, zero_bytes, s));
    const SlotTable<BPE> v{qf->table, tg.nslots};
    const uint32_t grid = (n + UPD_THREADS - 1) / UPD_THREADS;
    // a warp per listed unit or group, at most every key's
    const uint32_t lgrid = std::min<uint32_t>((n + LIST_THREADS / 32 - 1) / (LIST_THREADS / 32), (uint32_t)di.sms * 32);
    if (ins) {
        GQF_CK(cudaMemsetAsync(ib.seen, 0xFF, (size_t)hsize * 4, s));
        k_ins_stage<BPE><<<grid, UPD_THREADS, 0, s>>>(keys, n, v, tg.q, tg.r, ib, far);
        k_ins_sort<<<ib.nb, INS_THREADS, 0, s>>>(ib, far);
        k_ins_groups<BPE><<<ib.nb, INS_THREADS, 0, s>>>(v, ib, far);
        k_ins_apply<BPE><<<ib.nb, INS_THREADS, 0, s>>>(v, tg.r, ib, ar.err, far);
        k_ins_lists<BPE><<<lgrid, LIST_THREADS, 0, s>>>(v, tg.r, ib);
        count_launches(5);
    } else {
        k_del_locate<BPE><<<grid, UPD_THREADS, 0, s>>>(keys, n, v, tg.q, tg.r, claim, lead, far);
        k_del_apply<BPE><<<grid, UPD_THREADS, 0, s>>>(n, v, claim, lead, units, n_units, far);
        k_del_units<BPE><<<lgrid, LIST_THREADS, 0, s>>>(v, claim, units, n_units);
        count_launches(3);
    }
    GQF_CK(cudaGetLastError());
    if (fb) {
        f.far = far;
        f.keys = keys;
        f.n = n;
        f.nbytes = (uint32_t)tg.T;
        LayoutArgs &a = f.lay;
        a.A = BucketSrc{f.E, f.abase, 0, f.acnt};
        a.B = BucketSrc{f.bitems, f.bbase, 0, f.bcnt};
        a.table = qf->table;
        a.q = tg.q;
        a.r = tg.r;
        a.tb = FB_TB;
        a.nb = fnb;
        a.nslots = tg.nslots;
        a.op = op;
        a.nodup = ins ? 1 : 0;
        a.set_ok = 0;
        a.a_dups = nullptr;
        a.err = ar.err;
        // the most items a bucket's u16 counters allow (eight times its average)
        a.cap_items = 65520;
        const size_t smem = layout_smem_bytes(FB_TB, a.cap_items, BPE);
        GQF_CK(set_smem(k_update_fallback<BPE>, smem));
        // a quarter of the SMs: the launch must find room for all of its CTAs
        // at once beside other streams' kernels, and it rarely runs
        void *args[] = {&f};
        GQF_CK(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k_update_fallback<BPE>),
                                           dim3(std::max(1, di.sms / 4)), dim3(FB_THREADS), args, smem, s));
        count_launches(1);
    }
    return call_end(ar, s, ms);
}

template int local_update<1>(const gqf_sqf *, const uint32_t *, uint32_t, int, cudaStream_t, float *);
template int local_update<2>(const gqf_sqf *, const uint32_t *, uint32_t, int, cudaStream_t, float *);

}  // namespace gqf

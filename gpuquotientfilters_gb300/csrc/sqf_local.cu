// Cluster-local inserts and deletes, and the device-side rebuild behind
// queued updates.
#include "sqf_host.cuh"
#include "sqf_update.cuh"

namespace gqf {

// ------------------------------------------------------ rebuild on the device
template <int BPE>
int launch_fallback(FallbackArgs &f, const SqfGeom &tg, uint8_t *table, int op, int nodup, uint32_t *err,
                    cudaStream_t s, const BucketGeom *lists)
{
    f.nbytes = (uint32_t)tg.T;
    LayoutArgs &a = f.lay;
    a.A = BucketSrc{f.E, f.abase, 0, f.acnt};
    a.B = f.src2 ? BucketSrc{f.E2, f.bbase, 0, f.b2cnt} : BucketSrc{f.bitems, f.bbase, 0, f.bcnt};
    a.table = table;
    a.q = tg.q;
    a.r = tg.r;
    a.tb = lists ? lists->tb : FB_TB;
    a.nb = lists ? lists->nb : fallback_buckets(tg.q);
    f.lists_only = lists ? 1 : 0;
    a.nslots = tg.nslots;
    a.op = op;
    a.nodup = nodup;
    a.set_ok = 0;
    a.a_dups = nullptr;
    // a fix-up for every quotient: on an overfull table the spill passes
    // whole buckets (the extraction is done with Q by then)
    a.fix_list = f.Q;
    a.fix_cap = tg.nslots;
    a.err = err;
    a.cap_items = FB_CAP;
    size_t smem = layout_smem_bytes(FB_TB, a.cap_items, BPE);
    if (lists) smem = EXTRACT_TILE * sizeof(uint32_t);
    if (f.snap) smem = std::max(smem, set_update_smem(FB_TB, FB_THREADS, false));
    GQF_CK(set_smem(k_update_fallback<BPE>, smem));
    // one CTA per SM (two on large tables with small slots, whose layout is
    // the longest): the launch must find room for all of its CTAs at once
    // beside other streams' kernels
    const uint32_t work = std::max(a.nb, (tg.nslots + EXTRACT_TILE - 1) / EXTRACT_TILE);
    const uint32_t grid = std::min<uint32_t>(work, (uint32_t)device_info(current_device()).sms * (tg.q >= 24 ? 2 : 1));
    void *args[] = {&f};
    GQF_CK(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k_update_fallback<BPE>), dim3(grid),
                                       dim3(FB_THREADS), args, smem, s));
    count_launches(1);
    return GQF_OK;
}
template int launch_fallback<1>(FallbackArgs &, const SqfGeom &, uint8_t *, int, int, uint32_t *, cudaStream_t,
                                const BucketGeom *);
template int launch_fallback<2>(FallbackArgs &, const SqfGeom &, uint8_t *, int, int, uint32_t *, cudaStream_t,
                                const BucketGeom *);

// ------------------------------------------------------ cluster-local updates
struct LocalBufs {
    InsBatch ib;
    uint32_t hsize;
    uint32_t *far, *claim, *n_units;
    uint2 *units;
    uint4 *lead;
    FallbackArgs f;
    size_t zero_bytes;
};
// Control words and the delete's claims (zeroed) | the update's arrays or,
// when the rebuild behind them runs, that one's over them.
template <typename C>
static LocalBufs carve_local(C &c, const SqfGeom &tg, uint32_t n, bool ins, bool fallback)
{
    LocalBufs b{};
    InsBatch &ib = b.ib;
    // insert buckets of about 128 keys, one CTA each
    uint32_t lg = 0;
    while ((128ull << lg) < n && lg < std::min<uint32_t>(tg.q, 18)) lg++;
    ib.nb = 1u << lg;
    ib.shift = tg.q + tg.r - lg;
    const double avg = (double)n / ib.nb;
    ib.stride = (uint32_t)align_up((size_t)(avg + 10.0 * std::sqrt(avg) + 32.0), 32);
    b.hsize = 1024;
    while (b.hsize < 2ull * n) b.hsize <<= 1;
    ib.hmask = b.hsize - 1;
    FallbackArgs &f = b.f;
    b.far = c.template take<uint32_t>(1);
    f.bar = c.template take<uint32_t>(4, 16);
    f.fused_fail = c.template take<uint32_t>(1, 4);
    ib.n_over = c.template take<uint32_t>(1, 4);
    ib.pool = c.template take<uint32_t>(1, 4);
    b.n_units = ib.n_group = c.template take<uint32_t>(1, 4);
    if (ins) ib.cnt = c.template take<uint32_t>(ib.nb, 4);
    else b.claim = c.template take<uint32_t>(2 * ((tg.nslots + 31) / 32), 16);
    b.zero_bytes = c.off;
    const size_t at = c.off;
    if (ins) {
        ib.seen = c.template take<uint32_t>(b.hsize);
        ib.base = c.template take<uint32_t>(ib.nb);
        ib.key = c.template take<uint4>((size_t)ib.nb * ib.stride + n);
        ib.over = c.template take<uint4>(n);
    } else {
        b.lead = c.template take<uint4>(n);
        b.units = c.template take<uint2>(n);
    }
    if (fallback) {
        const size_t end = c.off;
        c.off = at;
        carve_fallback(c, f, tg, false);
        f.tiles = c.template take<Counts3>((tg.nslots + EXTRACT_TILE - 1) / EXTRACT_TILE + 1);
        f.Q = c.template take<uint32_t>(tg.nslots);
        f.E = c.template take<uint32_t>(tg.nslots);
        f.bitems = c.template take<uint32_t>(n);
        f.snap = tg.bpe == 1 && tg.q >= FB_TB ? c.template take<uint8_t>(tg.T) : nullptr;
        c.off = std::max(c.off, end);
    }
    return b;
}
size_t local_update_bytes(const SqfGeom &tg, uint32_t n, int op)
{
    Sizer z;
    carve_local(z, tg, n, op == OP_INSERT, true);
    return z.off;
}

template <int BPE>
int local_update(const gqf_sqf *qf, const uint32_t *keys, uint32_t n, int op, cudaStream_t s, float *ms, bool *far)
{
    const SqfGeom tg = geom_of(qf);
    const DeviceInfo &di = device_info(current_device());
    const bool ins = op == OP_INSERT, fallback = BPE == 2 || !ms;
    *far = false;
    Sizer z;
    carve_local(z, tg, n, ins, fallback);
    Arena &ar = arena(current_device(), s);
    std::lock_guard<std::mutex> lk(ar.mu);
    void *base = arena_reserve(ar, z.off);
    if (!base) return GQF_ERR_NOMEM;
    Carver c(base);
    LocalBufs b = carve_local(c, tg, n, ins, fallback);
    int st = call_begin(ar, s, ms != nullptr);
    if (st) return st;
    if (n == 0) return call_end(ar, s, ms);
    GQF_CK(cudaMemsetAsync(base, 0, b.zero_bytes, s));
    const SlotTable<BPE> v{qf->table, tg.nslots, walk_limit(tg.q)};
    const uint32_t grid = (n + UPD_THREADS - 1) / UPD_THREADS;
    // a warp per listed unit or group, at most every key's
    const uint32_t lgrid = std::min<uint32_t>((n + LIST_THREADS / 32 - 1) / (LIST_THREADS / 32), (uint32_t)di.sms * 32);
    if (ins) {
        InsBatch &ib = b.ib;
        GQF_CK(cudaMemsetAsync(ib.seen, 0xFF, (size_t)b.hsize * 4, s));
        k_ins_stage<BPE><<<grid, UPD_THREADS, 0, s>>>(keys, n, v, tg.q, tg.r, ib, b.far);
        k_ins_sort<<<ib.nb, INS_THREADS, 0, s>>>(ib, b.far);
        k_ins_groups<BPE><<<ib.nb, INS_THREADS, 0, s>>>(v, ib, b.far);
        k_ins_apply<BPE><<<ib.nb, INS_THREADS, 0, s>>>(v, tg.r, ib, ar.err, b.far);
        k_ins_lists<BPE><<<lgrid, LIST_THREADS, 0, s>>>(v, tg.r, ib);
        count_launches(5);
    } else {
        k_del_locate<BPE><<<grid, UPD_THREADS, 0, s>>>(keys, n, v, tg.q, tg.r, b.claim, b.lead, b.far);
        k_del_apply<BPE><<<grid, UPD_THREADS, 0, s>>>(n, v, b.claim, b.lead, b.units, b.n_units, b.far);
        k_del_units<BPE><<<lgrid, LIST_THREADS, 0, s>>>(v, b.claim, b.units, b.n_units);
        count_launches(3);
    }
    GQF_CK(cudaGetLastError());
    if (fallback) {
        FallbackArgs &f = b.f;
        f.gate = b.far;
        f.gate_bits = ~0u;
        f.src = f.snap ? f.snap : qf->table;
        f.keys = keys;
        f.n = n;
        st = launch_fallback<BPE>(f, tg, qf->table, op, ins ? 1 : 0, ar.err, s);
        return st ? st : call_end(ar, s, ms);
    }
    uint32_t rep[2];
    st = call_report(ar, s, b.far, rep);
    if (st) return st;
    GQF_CK(cudaEventElapsedTime(ms, ar.ev0, ar.ev1));
    *far = rep[1] != 0;
    return *far ? GQF_OK : dev_err_to_status(rep[0]);
}
template int local_update<1>(const gqf_sqf *, const uint32_t *, uint32_t, int, cudaStream_t, float *, bool *);
template int local_update<2>(const gqf_sqf *, const uint32_t *, uint32_t, int, cudaStream_t, float *, bool *);

template <int BPE>
static void load_local()
{
    load_kernels(k_ins_stage<BPE>, k_ins_groups<BPE>, k_ins_apply<BPE>, k_ins_lists<BPE>, k_del_locate<BPE>,
                 k_del_apply<BPE>, k_del_units<BPE>, k_update_fallback<BPE>);
}
void load_local_kernels()
{
    load_local<1>();
    load_local<2>();
    load_kernels(k_ins_sort);
}

}  // namespace gqf

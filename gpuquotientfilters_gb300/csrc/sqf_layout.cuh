// launch_layout: the bucket layouts of builds, merges and rebuilt tables.
// Instantiated for one slot size per translation unit (sqf_layout1.cu,
// sqf_layout2.cu).
#pragma once

#include "sqf_host.cuh"

namespace gqf {

template <int BPE>
int launch_layout(const LayoutPlan &p, const SqfGeom &tg, uint8_t *table, const BucketSrc &A, const BucketSrc &B,
                  int op, int nodup, bool set_ok, const uint32_t *a_dups, Scratch &sc, uint32_t *err, cudaStream_t s,
                  const uint32_t *gate)
{
    // slots past the last bucket's quotients only receive spill: clear them
    // (a gated launch leaves that to k_fallback_prepare)
    size_t tail = (size_t)(1u << tg.q) * BPE;
    if (!gate && tg.T > tail) GQF_CK(cudaMemsetAsync(table + tail, 0, tg.T - tail, s));
    LayoutArgs a;
    a.A = A;
    a.B = B;
    a.table = table;
    a.q = tg.q;
    a.r = tg.r;
    a.tb = p.g.tb;
    a.nb = p.g.nb;
    a.nslots = tg.nslots;
    a.cap_items = p.cap_items;
    a.op = op;
    a.nodup = nodup;
    a.set_ok = set_ok ? 1 : 0;
    a.a_dups = a_dups;
    a.status = sc.status;
    a.ticket = sc.ticket;
    a.fix_list = sc.fix_list;
    a.fix_cnt = sc.fix_cnt;
    a.fix_cap = sc.fix_cap;
    a.err = err;
    a.gate = gate;
    const int threads = (int)layout_threads(p.g.tb);
    const DeviceInfo &di = device_info(current_device());
    // (an empty launch costs its CTAs: a gated one takes what is resident)
    const uint32_t grid = gate ? std::min<uint32_t>(p.g.nb, (uint32_t)di.sms * 2) : p.g.nb;
    cudaError_t e = cudaSuccess;
    auto go = [&](auto kernel, size_t smem) {
        e = set_smem(kernel, smem);
        if (e == cudaSuccess) kernel<<<grid, threads, smem, s>>>(a);
    };
    if (BPE == 1 && set_ok) {
        const size_t smem = set_layout_smem(p.g.tb, threads);
        switch (p.g.tb) {
        case 15: go(k_set_layout<1024, 32>, smem); break;
        case 14: go(k_set_layout<512, 32>, smem); break;
        case 13: go(k_set_layout<256, 32>, smem); break;
        case 12: go(k_set_layout<256, 16>, smem); break;
        case 11: go(k_set_layout<128, 16>, smem); break;
        case 10: go(k_set_layout<128, 8>, smem); break;
        case 9: go(k_set_layout<64, 8>, smem); break;
        case 8: go(k_set_layout<32, 8>, smem); break;
        default: go(k_set_layout<32, 4>, smem); break;
        }
        GQF_CK(e);
        count_launches(1);
    }
    if ((op == OP_BUILD || op == OP_MERGE) && !set_ok && !gate) {
        // shared memory for a third more than the average bucket, as far as
        // the SM's goes (two-byte buckets of 32768 quotients); a larger one
        // keeps its remainders in the scratch
        a.rem_scratch = sc.rems;
        const double avg = (double)p.n_expect / p.g.nb;
        const size_t maxsm = (size_t)(di.smem_optin > 0 ? di.smem_optin : 99 * 1024) - 4096;  // less the static arrays
        const size_t fixed = group_layout_smem(p.g.tb, threads, BPE, 0);
        const size_t most = maxsm > fixed ? ((maxsm - fixed) / BPE) & ~(size_t)15 : 0;
        a.cap_items = (uint32_t)std::min(
            align_up((size_t)std::min(avg * 1.3 + 8.0 * std::sqrt(avg) + 64.0, 40000.0), 16), most);
        const size_t smem = group_layout_smem(p.g.tb, threads, BPE, a.cap_items);
        auto gg = [&](auto dup, auto uniq) {
            if (nodup) go(uniq, smem);
            else go(dup, smem);
        };
        switch (p.g.tb) {
        case 15: gg(k_group_layout<1024, 32, BPE, false>, k_group_layout<1024, 32, BPE, true>); break;
        case 14: gg(k_group_layout<512, 32, BPE, false>, k_group_layout<512, 32, BPE, true>); break;
        case 13: gg(k_group_layout<256, 32, BPE, false>, k_group_layout<256, 32, BPE, true>); break;
        case 12: gg(k_group_layout<256, 16, BPE, false>, k_group_layout<256, 16, BPE, true>); break;
        case 11: gg(k_group_layout<128, 16, BPE, false>, k_group_layout<128, 16, BPE, true>); break;
        case 10: gg(k_group_layout<128, 8, BPE, false>, k_group_layout<128, 8, BPE, true>); break;
        case 9: gg(k_group_layout<64, 8, BPE, false>, k_group_layout<64, 8, BPE, true>); break;
        case 8: gg(k_group_layout<32, 8, BPE, false>, k_group_layout<32, 8, BPE, true>); break;
        default: gg(k_group_layout<32, 4, BPE, false>, k_group_layout<32, 4, BPE, true>); break;
        }
        GQF_CK(e);
        count_launches(1);
    } else if (!set_ok || a_dups) {
        switch (p.g.tb) {
        case 15: go(k_bucket_layout<1024, 32, BPE>, p.smem); break;
        case 14: go(k_bucket_layout<512, 32, BPE>, p.smem); break;
        case 13: go(k_bucket_layout<256, 32, BPE>, p.smem); break;
        case 12: go(k_bucket_layout<256, 16, BPE>, p.smem); break;
        case 11: go(k_bucket_layout<128, 16, BPE>, p.smem); break;
        case 10: go(k_bucket_layout<128, 8, BPE>, p.smem); break;
        case 9: go(k_bucket_layout<64, 8, BPE>, p.smem); break;
        case 8: go(k_bucket_layout<32, 8, BPE>, p.smem); break;
        default: go(k_bucket_layout<32, 4, BPE>, p.smem); break;
        }
        GQF_CK(e);
        count_launches(1);
    }
    count_launches(1);
    k_fixup_occ<BPE><<<di.sms * 2, 256, 0, s>>>(table, sc.fix_list, sc.fix_cnt, sc.fix_cap, gate);
    GQF_CK(cudaGetLastError());
    return GQF_OK;
}

}  // namespace gqf

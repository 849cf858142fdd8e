// In-place merges, inserts and deletes of one-byte slots.
#include "sqf_host.cuh"

namespace gqf {

template <int THREADS, int QPT>
static cudaError_t launch_shape(const LayoutArgs &a, size_t smem, cudaStream_t s)
{
    auto kernel = a.src2              ? k_set_update<THREADS, QPT, UPDATE_TWO>
                  : a.op == OP_DELETE ? k_set_update<THREADS, QPT, UPDATE_DEL>
                                      : k_set_update<THREADS, QPT, UPDATE_ADD>;
    const cudaError_t e = set_smem(kernel, smem);
    if (e == cudaSuccess) kernel<<<a.nb, THREADS, smem, s>>>(a);
    return e;
}

// In-place update of one-byte slots: old contents from the snapshot (and
// `src2`), batch buckets of geometry p.
int launch_update(const LayoutPlan &p, const SqfGeom &tg, uint8_t *table, const uint8_t *src2,
                  const BucketSrc &B, int op, Scratch &sc, uint32_t *err, cudaStream_t s)
{
    const size_t tail = (size_t)1 << tg.q;
    if (tg.T > tail) GQF_CK(cudaMemsetAsync(table + tail, 0, tg.T - tail, s));
    LayoutArgs a;
    a.A = BucketSrc{nullptr, nullptr, 0, nullptr};
    a.B = B;
    a.table = table;
    a.q = tg.q;
    a.r = tg.r;
    a.tb = update_tb(tg.q);
    a.nb = 1u << (tg.q - a.tb);
    a.nslots = tg.nslots;
    a.cap_items = 0;
    a.op = op;
    a.nodup = 1;
    a.set_ok = 1;
    a.a_dups = nullptr;
    a.status = sc.status;
    a.ticket = sc.ticket;
    a.fix_list = sc.fix_list;
    a.fix_cnt = sc.fix_cnt;
    a.fix_cap = sc.fix_cap;
    a.err = err;
    a.src_table = sc.snap;
    a.src2 = src2;
    a.sub = p.g.tb - a.tb;
    a.fused_fail = sc.fused_fail;
    const int threads = (int)layout_threads(a.tb);
    const size_t smem = set_update_smem(a.tb, threads, src2 != nullptr);
    cudaError_t e = cudaSuccess;
    switch (a.tb) {
    case 13: e = launch_shape<256, 32>(a, smem, s); break;
    case 12: e = launch_shape<256, 16>(a, smem, s); break;
    case 11: e = launch_shape<128, 16>(a, smem, s); break;
    case 10: e = launch_shape<128, 8>(a, smem, s); break;
    case 9: e = launch_shape<64, 8>(a, smem, s); break;
    case 8: e = launch_shape<32, 8>(a, smem, s); break;
    default: e = launch_shape<32, 4>(a, smem, s); break;
    }
    GQF_CK(e);
    const DeviceInfo &di = device_info(current_device());
    k_fixup_occ<1><<<di.sms * 2, 256, 0, s>>>(table, sc.fix_list, sc.fix_cnt, sc.fix_cap);
    count_launches(2);
    GQF_CK(cudaGetLastError());
    return GQF_OK;
}

template <int THREADS, int QPT>
static void load_shape()
{
    load_kernels(k_set_update<THREADS, QPT, UPDATE_ADD>, k_set_update<THREADS, QPT, UPDATE_DEL>);
}
void load_inplace_kernels()
{
    load_shape<256, 32>();
    load_shape<256, 16>();
    load_shape<128, 16>();
    load_shape<128, 8>();
    load_shape<64, 8>();
    load_shape<32, 8>();
    load_shape<32, 4>();
}

}  // namespace gqf

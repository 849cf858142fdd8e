// C ABI of the standard quotient filter: host orchestration of the kernels.
#include "sqf_host.cuh"
#include "sqf_lookup.cuh"
#include "sqf_mirror.cuh"

namespace gqf {

// Bucket geometry for `n_expect` items over 2^q quotients: about 12k items
// per bucket (one CTA sorts a bucket in shared memory), at most 4096 buckets
// (the scatter keeps two u32 per bucket in shared memory).  `spread`: also
// enough buckets (of 256 quotients or more) that a small filter's layout uses
// every SM: 512 from q = 21 on, 256 below, where a launch and the look-back
// count for more (NoDup build, 512 against 256 buckets: q = 17 0.061 and
// 0.057 ms, q = 19 0.061 and 0.058, q = 21 0.058 and 0.060).
// `general`: k_bucket_layout may run.
static LayoutPlan plan_layout(uint32_t q, uint32_t r, uint64_t n_expect, uint64_t n_b_expect, bool general,
                              bool spread)
{
    const DeviceInfo &di = device_info(current_device());
    LayoutPlan p;
    uint32_t tb_lo = std::max<uint32_t>(7, q > 12 ? q - 12 : 0);
    uint32_t tb_hi = std::min<uint32_t>(q, 15);
    const uint32_t lg_spread = q >= 21 ? 9 : 8;
    if (spread) tb_hi = std::min(tb_hi, std::max<uint32_t>(q > lg_spread ? q - lg_spread : 0, std::min<uint32_t>(q, 8)));
    uint64_t denom = n_expect ? n_expect : 1;
    uint32_t tb = ceil_log2((12000ull << q) / denom);
    tb = std::min(std::max(tb, tb_lo), tb_hi);
    p.g.q = q;
    p.g.r = r;
    p.g.tb = tb;
    p.g.nb = 1u << (q - tb);
    p.g.shift = r + tb;
    p.g.fp_mask = (q + r >= 32) ? 0xFFFFFFFFu : ((1u << (q + r)) - 1u);
    double avg_b = (double)n_b_expect / p.g.nb;
    p.stride = (uint32_t)align_up((size_t)(avg_b + 10.0 * std::sqrt(avg_b) + 64.0), 32);
    p.n_expect = n_expect;
    p.cap_items = 0;
    p.smem = 0;
    if (!general) return p;
    int bpe = (r + 3) / 8;
    double avg = (double)n_expect / p.g.nb;
    uint32_t need = (uint32_t)(avg * 1.05 + 10.0 * std::sqrt(avg) + 256.0);
    size_t S = (size_t)1 << tb;
    size_t tile = tile_bytes(tb, bpe) + S / 8;
    size_t counters = 4 * (S / 2 + S / 32 + 8);
    size_t budget = 100 * 1024;
    size_t maxsm = (size_t)(di.smem_optin > 0 ? di.smem_optin : 99 * 1024) - 4096;
    if (counters + (size_t)need * bpe + tile + 16 > budget) budget = maxsm;
    size_t r0 = budget > tile + 16 ? budget - tile - 16 : 0;
    size_t cap = r0 > counters ? (r0 - counters) / bpe : 0;
    cap = std::min<size_t>(cap & ~(size_t)15, 65520);
    p.cap_items = (uint32_t)cap;
    p.smem = layout_smem_bytes(tb, p.cap_items, bpe);
    return p;
}

// Device-side exclusive scan of bucket counts into bases (nb <= 4096).
__global__ void __launch_bounds__(1024) k_scan_bases(const uint32_t *cnt, uint32_t nb, uint32_t *base)
{
    __shared__ uint32_t s[4097];
    __shared__ uint32_t sw[33];
    for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x) s[i] = cnt[i];
    __syncthreads();
    block_exclusive_scan_u32<1024>(s, nb, sw);
    for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x) base[i] = s[i];
}

// Extract a table's fingerprints (sorted for canonical tables) into E and
// bucket them by quotient range.  Count of elements stays on the device.
template <int BPE>
static int extract_into(const uint8_t *table, uint32_t nslots, size_t nbytes, uint32_t r, const BucketGeom &g,
                        Counts3 *tiles, uint32_t *Q, uint32_t *E, uint32_t *base, uint32_t *cnt, uint32_t *dups,
                        cudaStream_t s)
{
    uint32_t ntiles = (nslots + EXTRACT_TILE - 1) / EXTRACT_TILE;
    count_launches(6);
    k_tile_counts<BPE><<<ntiles, EXTRACT_THREADS, 0, s>>>(table, nslots, (uint32_t)nbytes, tiles, dups);
    k_scan_counts3<<<1, 1024, 0, s>>>(tiles, ntiles);
    k_occ_list<BPE><<<ntiles, EXTRACT_THREADS, 0, s>>>(table, nslots, (uint32_t)nbytes, tiles, Q);
    k_extract<BPE><<<ntiles, EXTRACT_THREADS, 0, s>>>(table, nslots, (uint32_t)nbytes, r, tiles, Q, E);
    uint32_t grid = (g.nb + 1 + 255) / 256;
    k_sorted_bounds<<<grid, 256, 0, s>>>(E, &tiles[ntiles].ne, g.nb, g.shift, base, cnt);
    k_bounds_to_counts<<<grid, 256, 0, s>>>(base, g.nb, cnt);
    GQF_CK(cudaGetLastError());
    return GQF_OK;
}

// Hash + bucket the batch keys.  exact: histogram + device scan first.
// Bucketing a batch: histogram + scan (exact bases) or speculative strides,
// then the scatter.  Batches of up to SMALL_BATCH keys (inserts, deletes,
// small builds) use 4096-key chunks so that enough CTAs share the work; the
// large ones 32K-key chunks.
constexpr uint32_t SMALL_BATCH = 1u << 22;
constexpr int SMALL_THREADS = 256, SMALL_IPT = 16;

template <int T, int IPT>
static int bucket_batch_keys(const uint32_t *keys, uint32_t n, const LayoutPlan &p, Scratch &sc, bool exact,
                             uint32_t *err, cudaStream_t s)
{
    const uint32_t grid = (n + T * IPT - 1) / (T * IPT);
    if (exact) {
        count_launches(2);
        GQF_CK(set_smem(k_bucket_hist<T, IPT>, p.g.nb * 4));
        k_bucket_hist<T, IPT><<<grid, T, p.g.nb * 4, s>>>(keys, n, p.g, sc.bcnt);
        k_scan_bases<<<1, 1024, 0, s>>>(sc.bcnt, p.g.nb, sc.bbase);
        GQF_CK(cudaMemsetAsync(sc.bcnt, 0, p.g.nb * 4, s));
    }
    count_launches(1);
    auto kfn = k_hash_bucket<T, IPT>;
    const size_t sm = (size_t)T * IPT * 4 + (size_t)p.g.nb * 8;
    GQF_CK(set_smem(kfn, sm));
    kfn<<<grid, T, sm, s>>>(keys, n, p.g, exact ? sc.bbase : nullptr, exact ? 0xFFFFFFFFu : p.stride, sc.bcnt,
                            sc.bitems, err);
    GQF_CK(cudaGetLastError());
    return GQF_OK;
}

static int bucket_batch(const uint32_t *keys, uint32_t n, const LayoutPlan &p, Scratch &sc, bool exact, uint32_t *err,
                        cudaStream_t s)
{
    if (n == 0) return GQF_OK;
    return n <= SMALL_BATCH ? bucket_batch_keys<SMALL_THREADS, SMALL_IPT>(keys, n, p, sc, exact, err, s)
                            : bucket_batch_keys<SCATTER_THREADS, SCATTER_IPT>(keys, n, p, sc, exact, err, s);
}

constexpr uint32_t ONE_LAUNCH_Q = 22;
constexpr uint32_t ONE_PASS_ITEMS = 1u << 20;
constexpr size_t SNAP_BESIDE = 16u << 20;  // table bytes from which a snapshot is copied on the side stream

// What a rebuild runs and needs: A = current contents of the table (unless it
// is a build), B = hashed batch keys or (two) the second table's contents.
struct Rebuild {
    bool needA, two;
    bool set_ok;    // the layout from lists has set semantics (see LayoutArgs::set_ok)
    bool in_place;  // one-byte slots, set semantics: decoded bucket by bucket from a snapshot
    bool exact;     // exact bucket bases from the start
    bool one_pass;  // the in-place batch in strides that hold all of it
    LayoutPlan p;
    ScratchReq spec, req;  // scratch with speculative bucket strides, and as it runs otherwise
    size_t bytes;
};
static Rebuild plan_rebuild(const SqfGeom &tg, uint32_t n, int op, int nodup, bool two, bool queued,
                            bool strides = true)
{
    Rebuild b{};
    b.needA = op != OP_BUILD;
    b.two = two;
    const bool update = op == OP_INSERT || op == OP_DELETE;
    b.set_ok = tg.r == 5 && (((op == OP_BUILD || op == OP_MERGE) && nodup) || op == OP_INSERT);
    b.in_place = tg.r == 5 && b.needA && (update || nodup);
    // A timed build uses speculative bucket strides (one pass over the keys)
    // and reruns with exact bucket bases if a bucket overflowed; the rerun
    // rewrites the whole table from the keys.  Updates read the table, so
    // they and all asynchronous calls bucket exactly.
    b.exact = op != OP_BUILD || queued;
    // expected items: the table holds at most nslots
    const uint64_t expect = std::min<uint64_t>((b.needA ? (uint64_t)(tg.nslots * 0.9) : 0) +
                                                   (two ? (uint64_t)(tg.nslots * 0.9) : n),
                                               (uint64_t)tg.nslots * 2);
    // an in-place update's batch keeps the large buckets (a layout bucket
    // reads its part of one); a build's are the layout's
    b.p = plan_layout(tg.q, tg.r, expect, two ? 0 : n, update || b.in_place, !b.in_place);
    b.req = ScratchReq{b.p.g.nb, std::max<size_t>(n, 1), b.needA, two, tg.nslots};
    // small filters are laid out in small buckets, which a nearly full table's
    // spill can pass whole
    b.req.every_fix = tg.q <= 22;
    if ((op == OP_BUILD || op == OP_MERGE) && !b.set_ok) b.req.rem_bytes = tg.bpe;
    b.spec = b.req;
    if (!two) b.spec.batch_items = (size_t)b.p.g.nb * b.p.stride;
    if (b.in_place) {
        // A small batch on a small table is bucketed in one pass, with room
        // for all of it in every bucket: three launches fewer than exact bases
        // need (a synchronous delete of 4096 keys at q = 15: 70 us, now 56).
        b.one_pass = strides && (uint64_t)b.p.g.nb * n <= ONE_PASS_ITEMS;
        if (b.one_pass) {
            b.p.stride = (uint32_t)align_up(n, 4);
            b.req.batch_items = std::max<size_t>((size_t)b.p.g.nb * b.p.stride, 1);
        }
        b.req.snap_bytes = tg.T;
        b.req.upd_nb = 1u << (tg.q - update_tb(tg.q));
        b.req.fallback = &tg;
    }
    carve(nullptr, b.req, true, &b.bytes);
    if (!b.exact) {
        size_t spec = 0;
        carve(nullptr, b.spec, true, &spec);
        b.bytes = std::max(b.bytes, spec);
    }
    return b;
}

template <int BPE>
static int rebuild(const gqf_sqf *qf, const gqf_sqf *qf2, const uint32_t *keys, uint32_t n, int op, int nodup,
                   cudaStream_t s, float *ms)
{
    const SqfGeom tg = geom_of(qf);
    Rebuild b = plan_rebuild(tg, n, op, nodup, qf2 != nullptr, ms == nullptr);
    const LayoutPlan &p = b.p;
    // duplicates in the table veto the set mode of an insert
    const bool insert = op == OP_INSERT;
    Arena &ar = arena(current_device(), s);
    std::lock_guard<std::mutex> lk(ar.mu);
    void *base = arena_reserve(ar, b.bytes);
    if (!base) return GQF_ERR_NOMEM;
    size_t bytes = 0;
    float ms_first = 0.0f;
    FallbackArgs behind{};
    // In-place update: the old contents are decoded bucket by bucket from a
    // snapshot of the table (no extraction pass, see LayoutArgs).  If a bucket
    // cannot be decoded (a table holding duplicate fingerprints, a run past
    // its slice), the op is done the general way from the snapshot: a
    // synchronous call decides on the host; behind an asynchronous one it is
    // queued, and does nothing unless the device-side failure flag is set.  On
    // tables up to ONE_LAUNCH_Q that is one cooperative launch; on larger ones
    // the layout is a launch of its own, which uses the whole GPU (q = 24,
    // overfull: 0.5 ms against 3.2).  A bucket that its shared memory cannot
    // sort (a fingerprint with tens of thousands of copies) is left to another
    // cooperative launch, which has more.
    if (b.in_place) {
        Scratch sc = carve(base, b.req, false, &bytes);
        int st = call_begin(ar, s, ms != nullptr);
        if (st) return st;
        // a large snapshot is copied on the side stream while the batch is
        // bucketed; a small one costs less than the two event waits
        const bool beside = n != 0 && tg.T > SNAP_BESIDE;
        if (beside) {
            cudaStream_t side = arena_side(ar);
            if (!side) return GQF_ERR_CUDA;
            GQF_CK(cudaEventRecord(ar.fork, s));
            GQF_CK(cudaStreamWaitEvent(side, ar.fork, 0));
            GQF_CK(cudaMemcpyAsync(sc.snap, qf->table, tg.T, cudaMemcpyDeviceToDevice, side));
            GQF_CK(cudaEventRecord(ar.join, side));
        } else {
            GQF_CK(cudaMemcpyAsync(sc.snap, qf->table, tg.T, cudaMemcpyDeviceToDevice, s));
        }
        GQF_CK(cudaMemsetAsync(sc.bcnt, 0, sc.ctrl_bytes, s));
        BucketSrc B{nullptr, nullptr, 0, nullptr};
        if (n) {
            st = bucket_batch(keys, n, p, sc, !b.one_pass, ar.err, s);
            if (st) return st;
            B = b.one_pass ? BucketSrc{sc.bitems, nullptr, p.stride, sc.bcnt} : BucketSrc{sc.bitems, sc.bbase, 0, sc.bcnt};
        }
        if (beside) GQF_CK(cudaStreamWaitEvent(s, ar.join, 0));
        // a filter merged with itself is read from the snapshot twice
        const uint8_t *src2 = !qf2 ? nullptr : qf2->table == qf->table ? sc.snap : qf2->table;
        st = launch_update(p, tg, qf->table, src2, B, op, sc, ar.err, s);
        if (st) return st;
        FallbackArgs &f = sc.fb;
        f.gate = sc.fused_fail;
        f.gate_bits = ~0u;
        f.src = sc.snap;
        f.src2 = src2;
        f.keys = keys;
        f.n = n;
        f.tiles = sc.tiles;
        f.Q = sc.Q;
        f.E = sc.E;
        f.E2 = sc.E2;
        f.bitems = sc.bitems;
        if (!ms) {
            if (tg.q > ONE_LAUNCH_Q) {
                FallbackArgs l = f;
                l.n = 0;
                l.lay.status = sc.status;
                l.lay.ticket = sc.ticket;
                l.lay.fix_cnt = sc.fix_cnt;
                l.abase = sc.abase;
                l.acnt = sc.acnt;
                l.bbase = sc.a2base;
                l.b2cnt = sc.a2cnt;
                st = launch_fallback<BPE>(l, tg, qf->table, op, nodup, ar.err, s, &p.g);
                if (st) return st;
                if (src2) B = BucketSrc{sc.E2, sc.a2base, 0, sc.a2cnt};
                st = launch_layout<BPE>(p, tg, qf->table, BucketSrc{sc.E, sc.abase, 0, sc.acnt}, B, op, nodup, false,
                                        nullptr, sc, ar.err, s, sc.fused_fail);
                if (st) return st;
                f.gate = ar.err;
                f.gate_bits = DEV_ERR_BUCKET_CAP;
            }
            st = launch_fallback<BPE>(f, tg, qf->table, op, nodup, ar.err, s);
            return st ? st : call_end(ar, s, nullptr);
        }
        uint32_t rep[2];
        st = call_report(ar, s, sc.fused_fail, rep);
        if (st) return st;
        GQF_CK(cudaEventElapsedTime(&ms_first, ar.ev0, ar.ev1));
        if (!rep[1]) {
            *ms = ms_first;
            return dev_err_to_status(rep[0]);
        }
        behind = f;
        GQF_CK(cudaMemcpyAsync(qf->table, sc.snap, tg.T, cudaMemcpyDeviceToDevice, s));
    }
    for (bool exact = b.exact;; exact = true) {
        Scratch sc = carve(base, exact ? b.req : b.spec, false, &bytes);
        int st = call_begin(ar, s, ms != nullptr);
        if (st) return st;
        GQF_CK(cudaMemsetAsync(sc.bcnt, 0, sc.ctrl_bytes, s));  // counters, look-back, ticket, fix-ups
        BucketSrc A{nullptr, nullptr, 0, nullptr}, B{nullptr, nullptr, 0, nullptr};
        if (b.needA) {
            st = extract_into<BPE>(qf->table, tg.nslots, tg.T, tg.r, p.g, sc.tiles, sc.Q, sc.E, sc.abase, sc.acnt,
                                   sc.a_dups, s);
            if (st) return st;
            A = BucketSrc{sc.E, sc.abase, 0, sc.acnt};
        }
        if (b.two) {
            st = extract_into<BPE>(qf2->table, tg.nslots, tg.T, tg.r, p.g, sc.tiles, sc.Q, sc.E2, sc.a2base, sc.a2cnt,
                                   nullptr, s);
            if (st) return st;
            B = BucketSrc{sc.E2, sc.a2base, 0, sc.a2cnt};
        } else if (n) {
            st = bucket_batch(keys, n, p, sc, exact, ar.err, s);
            if (st) return st;
            B = exact ? BucketSrc{sc.bitems, sc.bbase, 0, sc.bcnt} : BucketSrc{sc.bitems, nullptr, p.stride, sc.bcnt};
        }
        st = launch_layout<BPE>(p, tg, qf->table, A, B, op, nodup, b.set_ok, insert ? sc.a_dups : nullptr, sc, ar.err,
                                s);
        if (st) return st;
        if (!ms) return call_end(ar, s, nullptr);
        // synchronous: look at the error word before deciding
        uint32_t rep[2];
        st = call_report(ar, s, nullptr, rep);
        if (st) return st;
        if ((rep[0] & DEV_ERR_BUCKET_OVER) && !exact) continue;
        GQF_CK(cudaEventElapsedTime(ms, ar.ev0, ar.ev1));
        *ms += ms_first;
        if ((rep[0] & DEV_ERR_BUCKET_CAP) && b.in_place) {
            ms_first = *ms;
            behind.gate = ar.err;  // (holds the bit)
            behind.gate_bits = DEV_ERR_BUCKET_CAP;
            GQF_CK(cudaEventRecord(ar.ev0, s));
            st = launch_fallback<BPE>(behind, tg, qf->table, op, nodup, ar.err, s);
            if (st) return st;
            st = call_end(ar, s, ms);
            *ms += ms_first;
            return st;
        }
        return dev_err_to_status(rep[0]);
    }
}

// ------------------------------------------------------------- update routes
// Inserts and deletes of at most a key per 64 quotients on tables of 2^22
// quotients and more touch only the clusters they change (sqf_update.cuh);
// larger batches, and any on smaller tables, update the whole table in place,
// which costs the same at every fill.  A synchronous insert / delete in us,
// fill 0.8:
//               2^q / 1024 keys     2^q / 64           2^q / 16
//               local    in place   local     in place local      in place
//     q = 20    87/58    71/71      97/65     75/71    171/72     84/83
//     q = 22    88/65    110/110    115/76    111/110  252/107    116/114
//     q = 24    95/71    186/183    165/107   188/189  527/256    201/196
//     q = 26    104/79   551/552    372/276   569/568  1560/955   629/620
// and at fill 0.9 local ones of 2^q / 64 from q = 22 on take 221/127 (in place
// 113/110), 325/205 (192/188) and 592/476 (572/571).
//
// Two-byte slots (q <= 18) have no in-place form: all deletes, and inserts of
// at most a key per 16 quotients, are local.
static uint32_t local_max_keys(uint32_t q, uint32_t r, int op)
{
    if (r != 5) return op == OP_DELETE ? 0x7FFFFFFFu : 1u << (q - 4);
    return q >= 22 ? 1u << (q - 6) : 0u;
}

// Scratch bytes of an insert or delete of up to n keys, whichever way it goes.
static size_t update_scratch_bytes(const SqfGeom &tg, uint32_t n)
{
    size_t most = 0;
    // smaller batches may take the strides of one pass where this one does not
    const uint64_t buckets = 1ull << (tg.q - update_tb(tg.q));
    const size_t strides = tg.r == 5 ? 4 * std::min<uint64_t>(buckets * (n + 4ull), ONE_PASS_ITEMS + 4 * buckets) : 0;
    for (int op : {OP_INSERT, OP_DELETE}) {
        most = std::max(most, local_update_bytes(tg, std::min(n, local_max_keys(tg.q, tg.r, op)), op));
        for (bool queued : {false, true})
            most = std::max(most, plan_rebuild(tg, n, op, op == OP_INSERT, false, queued, false).bytes + strides);
    }
    return most;
}

template <int BPE>
static int update_t(const gqf_sqf *qf, const uint32_t *keys, uint32_t n, int op, cudaStream_t s, float *ms)
{
    float ms_local = 0.0f;
    if (n <= local_max_keys(qf->qbits, qf->rbits, op)) {  // (and empty batches)
        bool far = false;
        const int st = local_update<BPE>(qf, keys, n, op, s, ms, &far);
        if (st || !far) return st;
        ms_local = *ms;
    }
    const int st = rebuild<BPE>(qf, nullptr, keys, n, op, op == OP_INSERT ? 1 : 0, s, ms);
    if (ms) *ms += ms_local;
    return st;
}

// Sorted and unsorted lookups alike: results go to the queries' input positions
// either way (the reference sorts them back by index, quotientFilter.cu:
// 304-305), and probing the table in input order was faster than bucketing
// the queries first at every size (2^18 queries: 20 against 52 us at q = 22,
// 19 against 127 us at q = 26).
template <int BPE>
static int lookup_t(const gqf_sqf *qf, int n, const uint32_t *keys, uint32_t *out, cudaStream_t s, float *ms)
{
    const SqfGeom tg = geom_of(qf);
    Arena &ar = arena(current_device(), s);
    std::lock_guard<std::mutex> lk(ar.mu);
    // One-byte slots: transposing the table into the bit-plane mirror first
    // pays from one query per 32 slots and 768K queries on (2^19 queries: 26
    // us directly, 26 to 29 us through the mirror for q = 15 to 22; 2^20: 37
    // against 32 us).
    const bool mirror = BPE == 1 && (uint64_t)n * 32 >= tg.nslots && n >= (3 << 18);
    const TableView v{qf->table, tg.q, tg.r, tg.nslots, (uint32_t)tg.T, (uint32_t)(tg.T / 8)};
    const DeviceInfo &di = device_info(current_device());
    if (!mirror) {
        const int st = plain_begin(ar, s, ms != nullptr);
        if (st) return st;
        if (n > 0) {
            // one or two queries per thread: more threads in flight beat more
            // loads per thread for the dependent walks
            constexpr int QPT = BPE == 1 ? 2 : 1;
            const uint32_t per_block = LOOKUP_THREADS * QPT;
            const uint32_t grid = std::min<uint32_t>((n + per_block - 1) / per_block, (uint32_t)di.sms * 32);
            k_lookup_unsorted<BPE, QPT><<<grid, LOOKUP_THREADS, 0, s>>>(keys, (uint32_t)n, v, out);
            count_launches(1);
        }
        return plain_end(ar, s, ms);
    }
    uint4 *rec = static_cast<uint4 *>(arena_reserve(ar, mir_bytes(tg.nslots)));
    if (!rec) return GQF_ERR_NOMEM;
    GQF_CK(set_smem(k_sqf_mirror, 2 * (size_t)MIR_TILE));
    const int st = call_begin(ar, s, ms != nullptr);
    if (st) return st;
    const uint32_t ngroups = mir_groups(tg.nslots);
    const uint32_t ntiles = (uint32_t)(((uint64_t)(ngroups + 1) * MIR_SLOTS + MIR_TILE - 1) / MIR_TILE);
    k_sqf_mirror<<<std::min<uint32_t>(ntiles, (uint32_t)di.sms * 3), MIR_BUILD_THREADS, 2 * MIR_TILE, s>>>(
        v, rec, ngroups, ntiles, ar.err);
    const uint32_t grid = std::min<uint32_t>((n + MIR_LOOKUP_THREADS - 1) / MIR_LOOKUP_THREADS, (uint32_t)di.sms * 32);
    k_lookup_mirror<<<grid, MIR_LOOKUP_THREADS, 0, s>>>(keys, (uint32_t)n, v, rec, out);
    count_launches(2);
    return call_end(ar, s, ms);
}

void load_served_kernels()
{
    load_local_kernels();
    load_inplace_kernels();
    load_kernels(k_bucket_hist<SMALL_THREADS, SMALL_IPT>, k_hash_bucket<SMALL_THREADS, SMALL_IPT>,
                 k_bucket_hist<SCATTER_THREADS, SCATTER_IPT>, k_hash_bucket<SCATTER_THREADS, SCATTER_IPT>, k_scan_bases,
                 k_fixup_occ<1>, k_sqf_mirror, k_lookup_mirror, k_lookup_unsorted<1, 2>, k_lookup_unsorted<2, 1>);
}

// ------------------------------------------------ no-allocation bulk build
// Scratch for gqf_sqf_bulk_build_noalloc: a fixed array in the library's
// device image.  Host code must not use the symbol itself as an address;
// each device's address comes from cudaGetSymbolAddress on that device.
static __device__ __align__(256) unsigned char g_noalloc_scratch[GQF_NOALLOC_SCRATCH_BYTES];
// Per device: the array's device address (looked up on the first call, with
// that device current) and a mutex that serialises the calls on it.
struct NoallocDev {
    std::mutex mu;
    void *base = nullptr;
};
static std::mutex g_noalloc_map_mu;
static std::map<int, NoallocDev> g_noalloc_dev;

template <int BPE>
static int bulk_build_noalloc_t(const gqf_sqf *qf, uint32_t n, const uint32_t *keys, int nodup, cudaStream_t s)
{
    const int dev = current_device();
    NoallocDev *nd;
    {
        std::lock_guard<std::mutex> lk(g_noalloc_map_mu);
        nd = &g_noalloc_dev[dev];  // std::map nodes stay put
    }
    std::lock_guard<std::mutex> lk(nd->mu);
    if (!nd->base) {
        void *ptr = nullptr;
        GQF_CK(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
        nd->base = ptr;
    }
    char *base = static_cast<char *>(nd->base);
    const SqfGeom tg = geom_of(qf);
    const bool set_ok = tg.r == 5 && nodup;
    LayoutPlan p = plan_layout(tg.q, tg.r, n, n, false, false);  // few buckets: the fix-up list is small
    ScratchReq req{p.g.nb, std::max<size_t>(n, 1), false, false, tg.nslots};
    if (!set_ok) req.rem_bytes = BPE;
    size_t need = 0;
    carve(nullptr, req, true, &need);
    const size_t err_off = GQF_NOALLOC_SCRATCH_BYTES - 256;  // device error word
    if (need > err_off) return GQF_ERR_LIMIT;
    size_t got = 0;
    Scratch sc = carve(base, req, false, &got);
    uint32_t *err = reinterpret_cast<uint32_t *>(base + err_off);
    // the array keeps the previous call's contents: clear what starts at zero
    GQF_CK(cudaMemsetAsync(err, 0, sizeof(uint32_t), s));
    GQF_CK(cudaMemsetAsync(sc.bcnt, 0, sc.ctrl_bytes, s));
    BucketSrc A{nullptr, nullptr, 0, nullptr}, B{nullptr, nullptr, 0, nullptr};
    if (n) {
        int st = bucket_batch(keys, n, p, sc, true, err, s);
        if (st) return st;
        B = BucketSrc{sc.bitems, sc.bbase, 0, sc.bcnt};
    }
    int st = launch_layout<BPE>(p, tg, qf->table, A, B, OP_BUILD, nodup, set_ok, nullptr, sc, err, s);
    if (st) return st;
    uint32_t e = 0;
    GQF_CK(cudaMemcpyAsync(&e, err, sizeof(e), cudaMemcpyDeviceToHost, s));
    GQF_CK(cudaStreamSynchronize(s));
    return dev_err_to_status(e);
}

// One warp per bucket runs the build's look-back over host-given
// descriptors, with a caller-chosen poll limit (test support).
__global__ void k_lookback_probe(unsigned long long *status, uint32_t nb, uint32_t spin_limit, uint32_t *cin,
                                 uint32_t *err)
{
    const uint32_t b = blockIdx.x;
    if (b >= nb) return;
    const uint32_t c = lookback_cin_warp(status, b, err, spin_limit);
    if ((threadIdx.x & 31) == 0) cin[b] = c;
}

}  // namespace gqf

using namespace gqf;

#define BPE_DISPATCH(qf, fn, ...) (((qf)->rbits + 3) / 8 == 1 ? fn<1>(__VA_ARGS__) : fn<2>(__VA_ARGS__))

extern "C" {

size_t gqf_sqf_table_bytes(unsigned int q, unsigned int r)
{
    // calcNumSlotsGPU, quotientFilter.cu:37-42
    size_t table_bits = (size_t)(1u << q) * (r + 3);
    size_t table_slots = table_bits / 8;
    return (size_t)((double)table_slots * 1.1);
}

unsigned int gqf_sqf_num_slots(unsigned int q) { return (unsigned int)((double)(1u << q) * 1.1); }

size_t gqf_sqf_update_workspace_bytes(unsigned int q, unsigned int r, int n)
{
    if (!qr_ok(q, r) || n < 0) return 0;
    gqf_sqf f{};
    f.qbits = q;
    f.rbits = r;
    return align_up(update_scratch_bytes(geom_of(&f), (uint32_t)n), 1u << 20);
}

int gqf_sqf_init(gqf_sqf *qf, unsigned int q, unsigned int r)
{
    if (!qf || !qr_ok(q, r)) return GQF_ERR_ARG;
    qf->qbits = q;
    qf->rbits = r;
    qf->bytesPerElement = (r + 3) / 8;
    size_t T = gqf_sqf_table_bytes(q, r);
    unsigned char *t = nullptr;
    GQF_CK(cudaMalloc(&t, align_up(T, 256)));
    GQF_CK(cudaMemset(t, 0, align_up(T, 256)));
    qf->table = t;
    return GQF_OK;
}

int gqf_sqf_free(gqf_sqf *qf)
{
    if (!qf) return GQF_ERR_ARG;
    if (qf->table) GQF_CK(cudaFree(qf->table));
    qf->table = nullptr;
    return GQF_OK;
}

// the kernels read the table in aligned 8- and 16-byte words and bulk copies
static bool table_aligned(const void *t) { return (reinterpret_cast<uintptr_t>(t) & 15u) == 0; }
static bool sqf_ok(const gqf_sqf *qf)
{
    return qf && qf->table && table_aligned(qf->table) && qr_ok(qf->qbits, qf->rbits);
}

int gqf_sqf_bulk_build(const gqf_sqf *qf, int n, const uint32_t *d_keys, int no_duplicates, void *stream, float *ms)
{
    if (!sqf_ok(qf) || n < 0 || (n > 0 && !d_keys)) return GQF_ERR_ARG;
    return BPE_DISPATCH(qf, rebuild, qf, nullptr, d_keys, (uint32_t)n, OP_BUILD, no_duplicates ? 1 : 0,
                        static_cast<cudaStream_t>(stream), ms);
}

int gqf_sqf_bulk_build_noalloc(const gqf_sqf *qf, int n, const uint32_t *d_keys, int no_duplicates, void *stream)
{
    if (!sqf_ok(qf) || n < 0 || (n > 0 && !d_keys)) return GQF_ERR_ARG;
    if ((unsigned)n > GQF_NOALLOC_MAX_KEYS || qf->qbits > GQF_NOALLOC_MAX_Q) return GQF_ERR_LIMIT;
    return BPE_DISPATCH(qf, bulk_build_noalloc_t, qf, (uint32_t)n, d_keys, no_duplicates ? 1 : 0,
                        static_cast<cudaStream_t>(stream));
}

int gqf_sqf_insert(const gqf_sqf *qf, int n, const uint32_t *d_keys, void *stream, float *ms)
{
    if (!sqf_ok(qf) || n < 0 || (n > 0 && !d_keys)) return GQF_ERR_ARG;
    return BPE_DISPATCH(qf, update_t, qf, d_keys, (uint32_t)n, OP_INSERT, static_cast<cudaStream_t>(stream), ms);
}

int gqf_sqf_delete(const gqf_sqf *qf, int n, const uint32_t *d_keys, void *stream, float *ms)
{
    if (!sqf_ok(qf) || n < 0 || (n > 0 && !d_keys)) return GQF_ERR_ARG;
    return BPE_DISPATCH(qf, update_t, qf, d_keys, (uint32_t)n, OP_DELETE, static_cast<cudaStream_t>(stream), ms);
}

int gqf_sqf_insert_via_merge(const gqf_sqf *qf, const uint32_t *d_old, int n_old, const uint32_t *d_new, int n_new,
                             int no_duplicates, void *stream, float *ms)
{
    (void)d_old;
    (void)n_old;
    if (!sqf_ok(qf) || n_new < 0 || (n_new > 0 && !d_new)) return GQF_ERR_ARG;
    return BPE_DISPATCH(qf, rebuild, qf, nullptr, d_new, (uint32_t)n_new, OP_MERGE, no_duplicates ? 1 : 0,
                        static_cast<cudaStream_t>(stream), ms);
}

int gqf_sqf_merge(const gqf_sqf *qf1, const gqf_sqf *qf2, int no_duplicates, void *stream, float *ms)
{
    if (!sqf_ok(qf1) || !sqf_ok(qf2)) return GQF_ERR_ARG;
    if (qf1->qbits != qf2->qbits || qf1->rbits != qf2->rbits) return GQF_ERR_MISMATCH;
    return BPE_DISPATCH(qf1, rebuild, qf1, qf2, nullptr, 0u, OP_MERGE, no_duplicates ? 1 : 0,
                        static_cast<cudaStream_t>(stream), ms);
}

int gqf_sqf_lookup_unsorted(const gqf_sqf *qf, int n, const uint32_t *d_keys, uint32_t *d_out, void *stream, float *ms)
{
    if (!sqf_ok(qf) || n < 0 || (n > 0 && (!d_keys || !d_out))) return GQF_ERR_ARG;
    return BPE_DISPATCH(qf, lookup_t, qf, n, d_keys, d_out, static_cast<cudaStream_t>(stream), ms);
}

int gqf_sqf_lookup_sorted(const gqf_sqf *qf, int n, const uint32_t *d_keys, uint32_t *d_out, void *stream, float *ms)
{
    if (!sqf_ok(qf) || n < 0 || (n > 0 && (!d_keys || !d_out))) return GQF_ERR_ARG;
    return BPE_DISPATCH(qf, lookup_t, qf, n, d_keys, d_out, static_cast<cudaStream_t>(stream), ms);
}

int gqf_debug_lookback_probe(const unsigned long long *status, unsigned int nb, unsigned int spin_limit,
                             unsigned int *cin)
{
    if (!status || !cin || nb == 0 || nb > (1u << 20) || spin_limit == 0) return GQF_ERR_ARG;
    unsigned long long *d_status = nullptr;
    uint32_t *d_cin = nullptr, *d_err = nullptr;
    int st = GQF_OK;
    uint32_t e = 0;
    cudaError_t ce = cudaMalloc(&d_status, sizeof(unsigned long long) * nb);
    if (ce == cudaSuccess) ce = cudaMalloc(&d_cin, sizeof(uint32_t) * nb);
    if (ce == cudaSuccess) ce = cudaMalloc(&d_err, sizeof(uint32_t));
    if (ce == cudaSuccess) ce = cudaMemcpy(d_status, status, sizeof(unsigned long long) * nb, cudaMemcpyHostToDevice);
    if (ce == cudaSuccess) ce = cudaMemset(d_err, 0, sizeof(uint32_t));
    if (ce == cudaSuccess) {
        count_launches(1);
        k_lookback_probe<<<nb, 32>>>(d_status, nb, spin_limit, d_cin, d_err);
        ce = cudaGetLastError();
    }
    if (ce == cudaSuccess) ce = cudaDeviceSynchronize();
    if (ce == cudaSuccess) ce = cudaMemcpy(cin, d_cin, sizeof(uint32_t) * nb, cudaMemcpyDeviceToHost);
    if (ce == cudaSuccess) ce = cudaMemcpy(&e, d_err, sizeof(uint32_t), cudaMemcpyDeviceToHost);
    st = ce == cudaSuccess ? dev_err_to_status(e) : GQF_ERR_CUDA;
    cudaFree(d_status);
    cudaFree(d_cin);
    cudaFree(d_err);
    return st;
}

}  // extern "C"

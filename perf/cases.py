"""Performance cases of the quotient-filter engine.

Each case is one piece of work a program does through the public Python
entry points: building filters, querying them, updating them, merging them,
running a batch of many small ones.  Keys are uniform 32-bit words, like the
MT19937 draws of the benchmark configurations; lookups are half present and
half absent keys, shuffled.  Calls go to torch's current stream.  `sync`
says whether a case's calls wait for their result, as the reference's do
(each returns its device time), or are queued (sync=False), as a pipeline
or a server issues them.

Updates and merges change a table, so a pass first copies the base table
into a working table and then updates that copy: a service that prepares
the next version of a filter while readers still use the current one.
"""
import math
import random

import torch

import gpuquotientfilters_gb300 as G


def listed():
    return [
        # The smallest: one q=15 filter built, queried and thinned out with
        # synchronous calls (configuration 1).  Launches and latency.
        dict(name="sqf_step_q15", kind="step", q=15, r=5, n=19661, n_lookup=19661, n_delete=4096, sync=True),
        # The headline build: q=26 at fill 0.8, unique fingerprints.
        dict(name="sqf_build_q26", kind="build", q=26, r=5, n=53687091, nodup=True, sync=True),
        # A multiset build (every copy kept), queued, of a ragged size.
        dict(name="sqf_build_dup_q24", kind="build", q=24, r=5, n=12345677, nodup=False, sync=False),
        # Two-byte slots (13-bit remainders, low false-positive rate): build
        # and query.
        dict(name="sqf_wide_q18", kind="step", q=18, r=13, n=209715, n_lookup=262147, n_delete=0, sync=True),
        # The headline lookups: 2^24 unsorted queries on the q=26 filter.
        dict(name="sqf_lookup_q26", kind="lookup", q=26, r=5, n=53687091, n_lookup=1 << 24, sorted=False, sync=False),
        # The headline updates: 2^20 new keys in, 2^20 present keys out.
        dict(name="sqf_update_q26", kind="update", q=26, r=5, n=53687091, n_insert=1 << 20, n_delete=1 << 20,
             n_lookup=0, sync=True),
        # What a filter server issues (configuration 5's sizes): modest
        # insert, delete and lookup batches on a mid-sized filter, queued.
        dict(name="sqf_serve_q22", kind="update", q=22, r=5, n=2516582, n_insert=40009, n_delete=20011,
             n_lookup=100003, sync=False),
        # Two shards merged, then a key batch merged in.
        dict(name="sqf_merge_q22", kind="merge", q=22, r=5, n=1468006, n_other=1258291, n_new=300007, nodup=True,
             sync=True),
        # Many independent filters in one go (configuration 4): q 12..22,
        # fills 0.5..0.9, Pareto-sized lookups.
        dict(name="sqf_batch_256", kind="batch", filters=256, q_lo=12, q_hi=22, shapes=4),
        # Rank-and-select filter, 5-bit remainders: the q=26 build at fill 0.9
        # (configuration 3) and its 2^24 sorted lookups.
        dict(name="rsqf_build_q26", kind="rbuild", q=26, rbits=5, n=60397976),
        dict(name="rsqf_lookup_q26", kind="rlookup", q=26, rbits=5, n=60397976, n_lookup=1 << 24, sorted=True,
             sync=False),
        # Rank-and-select filter, 8-bit remainders: an incremental batch into
        # a filter at fill 0.9.
        dict(name="rsqf_insert_q23_r8", kind="rinsert", q=23, rbits=8, n=7549747, n_insert=1 << 17),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "build", "lookup", "update", "merge", "batch", "rbuild", "rlookup", "rinsert"])
    sync = rng.random() < 0.5
    if kind == "batch":
        lo = rng.randint(12, 17)
        return dict(kind=kind, filters=_log_int(rng, 16, 256), q_lo=lo, q_hi=rng.randint(lo, 22),
                    shapes=rng.randrange(1 << 20))
    if kind in ("rbuild", "rlookup", "rinsert"):
        rbits = rng.choice([5, 8])
        q = rng.randint(15, 26 if rbits == 5 else 23)
        n = int(rng.uniform(0.5, 0.9) * (1 << q))
        if kind == "rbuild":
            return dict(kind=kind, q=q, rbits=rbits, n=n)
        if kind == "rlookup":
            return dict(kind=kind, q=q, rbits=rbits, n=n, n_lookup=_log_int(rng, 1 << 10, 1 << 24),
                        sorted=rng.random() < 0.5, sync=sync)
        return dict(kind=kind, q=q, rbits=rbits, n=n, n_insert=_log_int(rng, 256, max(257, (1 << q) // 64)))
    if kind == "step":
        r = rng.choice([5, 13])
        q = rng.randint(12, 18)
        n = int(rng.uniform(0.3, 0.9) * (1 << q))
        return dict(kind=kind, q=q, r=r, n=n, n_lookup=_log_int(rng, 256, 1 << 19),
                    n_delete=rng.randint(0, n // 4), sync=sync)
    q = rng.randint(16, 26)
    n = int(rng.uniform(0.4, 0.9) * (1 << q))
    if kind == "build":
        return dict(kind=kind, q=q, r=5, n=min(n, 53687091), nodup=rng.random() < 0.7, sync=sync)
    if kind == "lookup":
        return dict(kind=kind, q=q, r=5, n=n, n_lookup=_log_int(rng, 1 << 10, 1 << 24), sorted=rng.random() < 0.5,
                    sync=sync)
    if kind == "update":
        n = min(n, int(0.85 * (1 << q)))
        return dict(kind=kind, q=q, r=5, n=n, n_insert=_log_int(rng, 256, (1 << q) // 16),
                    n_delete=_log_int(rng, 256, (1 << q) // 16), n_lookup=_log_int(rng, 256, 1 << 20), sync=sync)
    q = min(q, 24)
    part = (1 << q) // 2
    return dict(kind=kind, q=q, r=5, n=int(rng.uniform(0.3, 0.8) * part), n_other=int(rng.uniform(0.3, 0.8) * part),
                n_new=_log_int(rng, 256, part // 8), nodup=rng.random() < 0.7, sync=sync)


# --------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _keys(g, n):
    k = torch.randint(0, 1 << 32, (n,), dtype=torch.int64, device="cuda", generator=g)
    return torch.where(k >= 1 << 31, k - (1 << 32), k).to(torch.int32)


def _queries(g, keys, n):
    """Half present keys, half fresh ones, shuffled."""
    half = n // 2
    pos = keys[torch.randint(0, keys.numel(), (half,), device="cuda", generator=g)]
    q = torch.cat([pos, _keys(g, n - half)])
    return q[torch.randperm(n, device="cuda", generator=g)].contiguous()


def _batch_shapes(case):
    rng = random.Random(case["shapes"])
    out = []
    for _ in range(case["filters"]):
        q = rng.randint(case["q_lo"], case["q_hi"])
        n = int(rng.uniform(0.5, 0.9) * (1 << q))
        nl = int(min(max(rng.paretovariate(1.5) * 256.0, 256), 1 << 20))
        out.append((q, n, nl))
    return out


def _inputs(case, seed):
    """Every key array of a case, from the seed alone."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "batch":
        return [(lambda k: dict(keys=k, lookups=_queries(g, k, nl)))(_keys(g, n)) for _, n, nl in _batch_shapes(case)]
    d = dict(keys=_keys(g, case["n"]))
    if case.get("n_lookup"):
        d["lookups"] = _queries(g, d["keys"], case["n_lookup"])
    if case.get("n_delete"):
        d["deletes"] = d["keys"][: case["n_delete"]].clone()
    if case.get("n_insert"):
        d["inserts"] = _keys(g, case["n_insert"])
    if kind == "merge":
        d["other"] = _keys(g, case["n_other"])
        d["new"] = _keys(g, case["n_new"])
    return d


# --------------------------------------------------------------- geometry
def _table_bytes(q, r):
    return int(((1 << q) * (r + 3) // 8) * 1.1)


def _padded(q, r):
    return (_table_bytes(q, r) + 255) // 256 * 256


def _num_slots(q):
    return int((1 << q) * 1.1)


def _rsqf_bytes(q, rbits):
    blocks = ((1 << q) + 63) // 64 + 1
    return blocks, (blocks + 1) * (17 + 8 * rbits)


def _sqf(q, r):
    """A filter whose table is a torch tensor."""
    t = torch.zeros(_padded(q, r), dtype=torch.uint8, device="cuda")
    return G.quotient_filter(q, r, (r + 3) // 8, t.data_ptr()), t[: _table_bytes(q, r)]


def _rsqf(q, rbits):
    blocks, nbytes = _rsqf_bytes(q, rbits)
    t = torch.zeros(nbytes + 16, dtype=torch.uint8, device="cuda")  # 16 spare bytes, as initCQFGPU allocates
    f = G.countingQuotientFilterGPU(q, blocks, t.data_ptr())
    f._rbits = rbits
    return f, t[:nbytes]


def _results(n):
    return torch.empty(n, dtype=torch.int32, device="cuda")


# --------------------------------------------------------------- prepare / run
def prepare(case, seed):
    kind = case["kind"]
    d = _inputs(case, seed)
    s = torch.cuda.current_stream()
    st = dict(case=case)
    if kind == "batch":
        # one buffer for all tables, one for all results
        shapes = _batch_shapes(case)
        st["tables"] = torch.zeros(sum(_padded(q, 5) for q, _, _ in shapes), dtype=torch.uint8, device="cuda")
        st["out"] = _results(sum(nl for _, _, nl in shapes))
        jobs, t0, o0 = [], 0, 0
        for (q, _, nl), x in zip(shapes, d):
            f = G.quotient_filter(q, 5, 1, st["tables"].data_ptr() + t0)
            jobs.append((f, x["keys"], x["lookups"], st["out"][o0: o0 + nl]))
            t0, o0 = t0 + _padded(q, 5), o0 + nl
        st.update(batch=G.Batch(jobs), jobs=jobs)
        return st
    st.update(d)
    if "lookups" in d:
        st["out"] = _results(d["lookups"].numel())
    if kind in ("rbuild", "rlookup", "rinsert"):
        st["f"], st["table"] = _rsqf(case["q"], case["rbits"])
        st["ret"] = _results(case["n_insert"] if kind == "rinsert" else case["n"])
        if kind != "rbuild":
            G.insertGPU(st["f"], case["n"], d["keys"], _results(case["n"]), stream=s)
        if kind == "rinsert":
            st["base"] = st["table"].clone()
        return st
    q, r = case["q"], case["r"]
    st["f"], st["table"] = _sqf(q, r)
    if kind in ("lookup", "update", "merge"):
        G.bulkBuildSegmentedLayouts(st["f"], case["n"], d["keys"], case.get("nodup", True), stream=s)
    if kind in ("update", "merge"):
        st["base"] = st["table"].clone()
    if kind == "merge":
        st["f2"], st["table2"] = _sqf(q, r)
        G.bulkBuildSegmentedLayouts(st["f2"], case["n_other"], d["other"], case["nodup"], stream=s)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    s = torch.cuda.current_stream()
    if kind == "batch":
        st["batch"].run(stream=s)
        return {"tables": st["tables"], "slots": st["out"]}
    f, table = st["f"], st["table"]
    sync = case.get("sync", True)
    if kind == "rbuild":
        table.zero_()
        G.insertGPU(f, case["n"], st["keys"], st["ret"], stream=s)
        return {"blocks": table, "slots": st["ret"]}
    if kind == "rinsert":
        table.copy_(st["base"])
        G.insertGPU(f, case["n_insert"], st["inserts"], st["ret"], stream=s)
        return {"blocks": table, "slots": st["ret"]}
    if kind == "rlookup":
        op = G.launchLookups if case["sorted"] else G.launchUnsortedLookupsRSQF
        op(f, case["n_lookup"], st["lookups"], st["out"], stream=s, sync=sync)
        return {"slots": st["out"]}
    if kind == "lookup":
        op = G.launchSortedLookups if case["sorted"] else G.launchUnsortedLookups
        op(f, case["n_lookup"], st["lookups"], st["out"], stream=s, sync=sync)
        return {"slots": st["out"]}
    if kind == "build":
        G.bulkBuildSegmentedLayouts(f, case["n"], st["keys"], case["nodup"], stream=s, sync=sync)
        return {"table": table}
    if kind == "step":
        G.bulkBuildSegmentedLayouts(f, case["n"], st["keys"], True, stream=s, sync=sync)
        G.launchUnsortedLookups(f, case["n_lookup"], st["lookups"], st["out"], stream=s, sync=sync)
        if case["n_delete"]:
            G.superclusterDeletes(f, case["n_delete"], st["deletes"], stream=s, sync=sync)
        return {"table": table, "slots": st["out"]}
    table.copy_(st["base"])
    if kind == "update":
        G.insert(f, case["n_insert"], st["inserts"], stream=s, sync=sync)
        G.superclusterDeletes(f, case["n_delete"], st["deletes"], stream=s, sync=sync)
        if not case["n_lookup"]:
            return {"table": table}
        G.launchSortedLookups(f, case["n_lookup"], st["lookups"], st["out"], stream=s, sync=sync)
        return {"table": table, "slots": st["out"]}
    G.mergeTwoFilters(f, st["f2"], case["nodup"], stream=s, sync=sync)
    G.insertViaMerge(f, st["keys"], case["n"], st["new"], case["n_new"], case["nodup"], stream=s, sync=sync)
    return {"table": table}


# --------------------------------------------------------------- work
def work(case):
    """Bytes a pass cannot do without: every key, base table and result once.
    Lookups read the table once, or one 32-byte sector a query where that is
    less.  The arithmetic is integer hashing and bit work: no flops."""
    kind = case["kind"]

    def probe(n, table):
        return 8 * n + min(table, 32 * n)

    if kind == "batch":
        b = sum(4 * n + _table_bytes(q, 5) + probe(nl, _table_bytes(q, 5)) for q, n, nl in _batch_shapes(case))
        return {"bytes": b, "flops": 0}
    if kind[0] == "r":
        t = _rsqf_bytes(case["q"], case["rbits"])[1]
        b = {"rbuild": 8 * case["n"] + t, "rlookup": probe(case.get("n_lookup", 0), t),
             "rinsert": 8 * case.get("n_insert", 0) + 2 * t}[kind]
        return {"bytes": b, "flops": 0}
    t = _table_bytes(case["q"], case["r"])
    nl = case.get("n_lookup", 0)
    if kind == "build":
        b = 4 * case["n"] + t
    elif kind == "lookup":
        b = probe(nl, t)
    elif kind == "step":
        b = 4 * (case["n"] + case["n_delete"]) + t + probe(nl, t)
    elif kind == "update":
        b = 2 * t + 4 * (case["n_insert"] + case["n_delete"]) + probe(nl, t)
    else:
        b = 3 * t + 4 * case["n_new"]
    return {"bytes": b, "flops": 0}


# --------------------------------------------------------------- exact
def _fingerprints(keys, q, r):
    """Normal_APHash of the keys, modulo 2^(q + r), in 64-bit arithmetic."""
    m32 = 0xFFFFFFFF
    v = keys.to(torch.int64) & m32
    h = torch.full_like(v, 0xAAAAAAAA)
    for i, sh in enumerate((24, 16, 8, 0)):
        c = (v >> sh) & 0xFF
        if i & 1:
            h = h ^ ((((h << 11) & m32) ^ c ^ (h >> 5)) ^ m32)
        else:
            h = h ^ ((h << 7) & m32) ^ c ^ (h >> 3)
    return h & ((1 << (q + r)) - 1)


def _layout(fps, q, r):
    """Slots and table bytes of sorted fingerprints: each item goes to the
    first slot at or after its quotient that the items before it left free."""
    n = fps.numel()
    quot = fps >> r
    idx = torch.arange(n, dtype=torch.int64, device="cuda")
    pos = idx + torch.cummax(quot - idx, 0).values if n else idx
    cont = torch.zeros(n, dtype=torch.int64, device="cuda")
    cont[1:] = (quot[1:] == quot[:-1]).to(torch.int64)
    slots = torch.zeros(_num_slots(q), dtype=torch.int64, device="cuda")
    slots[pos] = ((fps & ((1 << r) - 1)) << 3) | (cont << 1) | (pos != quot).to(torch.int64)
    slots[torch.unique_consecutive(quot)] |= 4
    bpe = (r + 3) // 8
    table = torch.zeros(_table_bytes(q, r), dtype=torch.uint8, device="cuda")
    for b in range(bpe):
        table[b: slots.numel() * bpe: bpe] = ((slots >> (8 * (bpe - 1 - b))) & 0xFF).to(torch.uint8)
    return pos, table


def _find(fps, pos, want):
    """Slot of the first stored copy of each wanted fingerprint, or -1."""
    if not fps.numel():
        return torch.full((want.numel(),), -1, dtype=torch.int32, device="cuda")
    i = torch.searchsorted(fps, want).clamp(max=fps.numel() - 1)
    return torch.where(fps[i] == want, pos[i], torch.full_like(i, -1)).to(torch.int32)


def exact(case, seed):
    """The same outputs from the sorted fingerprints.  The rank-and-select
    filter's layout depends on the order its items went in, so its outputs
    have no such closed form."""
    kind = case["kind"]
    if kind[0] == "r":
        return None
    d = _inputs(case, seed)
    if kind == "batch":
        tables, slots = [], []
        for (q, _, _), x in zip(_batch_shapes(case), d):
            fps = torch.unique(_fingerprints(x["keys"], q, 5))
            pos, t = _layout(fps, q, 5)
            tables.append(torch.nn.functional.pad(t, (0, _padded(q, 5) - t.numel())))
            slots.append(_find(fps, pos, _fingerprints(x["lookups"], q, 5)))
        return {"tables": torch.cat(tables), "slots": torch.cat(slots)}
    q, r = case["q"], case["r"]
    fps = _fingerprints(d["keys"], q, r)
    nodup = case.get("nodup", True)
    if kind == "merge":
        parts = [torch.unique(p) if nodup else p for p in (fps, _fingerprints(d["other"], q, r))]
        fps = torch.cat(parts + [_fingerprints(d["new"], q, r)])
    fps = torch.unique(fps) if nodup else torch.sort(fps).values
    want = _fingerprints(d["lookups"], q, r) if "lookups" in d else None
    slots = None
    if kind == "step":  # lookups come before the deletes
        slots = _find(fps, _layout(fps, q, r)[0], want)
    if "inserts" in d:
        fps = torch.unique(torch.cat([fps, _fingerprints(d["inserts"], q, r)]))
    if "deletes" in d:
        fps = fps[~torch.isin(fps, _fingerprints(d["deletes"], q, r))]
    pos, table = _layout(fps, q, r)
    if want is not None and slots is None:
        slots = _find(fps, pos, want)
    if kind == "lookup":
        return {"slots": slots}
    return {"table": table} if slots is None else {"table": table, "slots": slots}

"""Cluster-local inserts and deletes on the GPU, at the sizes and fills where
they can go wrong: whole tables compared with the oracle byte for byte."""
import numpy as np
import pytest

import oracle as O
from conftest import to_dev

pytestmark = pytest.mark.gpu


def check(G, f, q, r, t):
    raw = G.table_bytes(f)
    if not np.array_equal(raw, t):
        d = np.nonzero(raw != t)[0]
        raise AssertionError("%d bytes differ, first at %d" % (d.size, d[0]))


def ops(G, torch, q, r, keys, nodup, batches, sync):
    """Builds, then applies (op, keys) one after the other beside the oracle."""
    f = G.initFilterGPU(q, r)
    t = O.sqf_new(q, r)
    try:
        G.bulkBuildSegmentedLayouts(f, keys.size, to_dev(torch, keys), nodup)
        assert O.sqf_bulk_build(t, q, r, keys, nodup) == 0
        for op, k in batches:
            d = to_dev(torch, k)
            (G.insert if op == "insert" else G.superclusterDeletes)(f, k.size, d, sync=sync)
            if not sync:
                G.stream_status()
            (O.sqf_insert if op == "insert" else O.sqf_delete)(t, q, r, k)
            check(G, f, q, r, t)
    finally:
        G.freeFilterGPU(f)


@pytest.mark.parametrize("sync", [True, False])
@pytest.mark.parametrize("q,r,alpha,nodup", [
    (7, 5, 0.7, True), (8, 5, 1.0, True), (12, 5, 1.03, True),       # whole table within one walk
    (13, 5, 0.9, False), (16, 5, 0.85, True), (18, 5, 0.9, False),   # ordinary, repeated fingerprints
    (16, 5, 1.04, True), (15, 13, 1.05, True), (16, 5, 1.05, False), # nearly full: stretches past the walk limit
    (14, 13, 0.8, True), (17, 13, 0.9, False),                       # two-byte slots
    (20, 5, 0.02, True), (20, 5, 0.6, True),                         # sparse
])
def test_local_updates(gqf, cuda, q, r, alpha, nodup, sync):
    n = int(alpha * (1 << q))
    keys = O.mt_keys(300 + q, n)
    m = max(1, (1 << q) // 16)  # the largest local insert
    free = O.sqf_num_slots(q) - n
    new = O.mt_keys(301 + q, 4 * m)
    small = new[: max(1, min(m, free // 2))]
    batches = [
        ("delete", np.concatenate([keys[:m], keys[: m // 2], new[:7]])),  # repeats, absent keys
        ("insert", small),
        ("insert", np.concatenate([small[::3], keys[-m // 3:]])[:m]),     # mostly stored already
        ("delete", np.concatenate([small[1::2], keys[m: 3 * m]])),
        ("insert", np.repeat(new[m: m + max(1, m // 8)], 8)[:m]),         # every key several times
        ("delete", keys),                                                 # everything
        ("insert", new[:m]),
    ]
    ops(gqf, cuda, q, r, keys, nodup, batches, sync)


def test_local_insert_one_hot_key_and_narrow_range(gqf, cuda):
    """A batch that is mostly one key, and one whose keys all fall in a few
    quotients' range (groups past their region and past shared memory)."""
    q, r = 18, 5
    keys = O.mt_keys(400, int(0.5 * (1 << q)))
    m = (1 << q) // 16
    hot = np.concatenate([np.full(m - 500, 12345, np.uint32), O.mt_keys(401, 500)])
    cand = O.mt_keys(402, 1 << 21)
    narrow = cand[(O.aphash(cand, q, r) >> r) < 2600][:m]
    assert narrow.size > 8000
    ops(gqf, cuda, q, r, keys, True, [("insert", hot), ("insert", narrow), ("delete", narrow[::2])], True)


@pytest.mark.parametrize("q", [10, 14, 17])
def test_local_insert_past_capacity_is_full(gqf, cuda, q):
    r = 5
    n = int(1.05 * (1 << q))
    f = gqf.initFilterGPU(q, r)
    try:
        k = O.mt_keys(500 + q, 4 * n)
        u = k[np.sort(np.unique(O.aphash(k, q, r), return_index=True)[1])]  # distinct fingerprints
        gqf.bulkBuildSegmentedLayouts(f, n, to_dev(cuda, u[:n]), True)
        with pytest.raises(gqf.GQFError) as e:
            at = n
            for _ in range(40):
                m = (1 << q) // 16
                gqf.insert(f, m, to_dev(cuda, u[at: at + m]))
                at += m
        assert e.value.status == gqf.GQF_ERR_FULL
    finally:
        gqf.freeFilterGPU(f)

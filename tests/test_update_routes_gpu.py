"""Inserts and deletes on both sides of the lines between their routes: the
cluster-local update, the in-place one, and the rebuild behind either (tables
with copies, long clusters, a fingerprint with more copies than the rebuild's
first form can sort), queued and synchronous; whole tables against the oracle."""
import numpy as np
import pytest

import oracle as O
from conftest import to_dev
from sqf_model import Contents, check

pytestmark = pytest.mark.gpu


def apply(G, torch, f, c, op, keys, sync):
    (G.insert if op == "insert" else G.superclusterDeletes)(f, keys.size, to_dev(torch, keys), sync=sync)
    G.stream_status()
    (c.insert if op == "insert" else c.delete)(keys)
    check(G, f, c.table(), "%s of %d" % (op, keys.size))


@pytest.mark.parametrize("sync", [True, False])
@pytest.mark.parametrize("q,r,fill,nodup", [
    (7, 5, 0.6, True), (7, 5, 0.6, False), (9, 5, 0.8, False), (10, 13, 0.9, False), (12, 5, 0.9, True),
    (12, 13, 1.0, True), (13, 5, 0.7, False), (14, 5, 0.95, True), (17, 5, 0.9, False), (21, 5, 0.5, True),
    (22, 5, 0.8, True), (22, 5, 0.95, True), (22, 5, 0.4, False), (23, 5, 0.3, True), (23, 5, 0.3, False)])
def test_update_routes(gqf, cuda, q, r, fill, nodup, sync):
    n = int(fill * (1 << q))
    keys = O.mt_keys(1000 + q, n)
    if not nodup:
        keys = np.concatenate([keys[: n - n // 8], keys[: n // 8]])
    line = max(1, (1 << q) // 64)  # the largest local batch from q = 22 on
    new = O.mt_keys(1001 + q, 2 * line + 7)
    room = max(1, (O.sqf_num_slots(q) - n) // 2)
    f, c = gqf.initFilterGPU(q, r), Contents(q, r, keys, nodup)
    try:
        gqf.bulkBuildSegmentedLayouts(f, keys.size, to_dev(cuda, keys), nodup)
        apply(gqf, cuda, f, c, "delete", np.concatenate([keys[: line // 2], new[: line // 2 + 1]]), sync)
        apply(gqf, cuda, f, c, "insert", new[: min(line, room)], sync)
        apply(gqf, cuda, f, c, "delete", keys[:line], sync)
        apply(gqf, cuda, f, c, "delete", np.concatenate([keys[line: 2 * line + 1], keys[:3]]), sync)
        apply(gqf, cuda, f, c, "insert", new[: min(line + 1, room)], sync)
        apply(gqf, cuda, f, c, "delete", keys[n // 2:], sync)
        apply(gqf, cuda, f, c, "insert", np.concatenate([keys[n // 2: n // 2 + 4 * line], new[:9], new[:9]]), sync)
    finally:
        gqf.freeFilterGPU(f)


@pytest.mark.parametrize("sync", [True, False])
@pytest.mark.parametrize("q", [16, 23])
def test_update_of_a_bucket_too_large_for_the_steps(gqf, cuda, q, sync):
    r, copies = 5, 31000
    cand = O.mt_keys(1049, 1000)
    hot = cand[(O.aphash(cand, q, r) >> r) < (1 << q) // 4][0]  # its copies fit the slots behind it
    keys = np.concatenate([np.full(copies, hot, np.uint32), O.mt_keys(1050 + q, (1 << q) // 4)])
    f, c = gqf.initFilterGPU(q, r), Contents(q, r, keys, False)
    try:
        gqf.bulkBuildSegmentedLayouts(f, keys.size, to_dev(cuda, keys), False)
        many = np.concatenate([np.full(copies - 5, hot, np.uint32), keys[copies: copies + (1 << q) // 64]])
        apply(gqf, cuda, f, c, "insert", np.concatenate([keys[-100:], O.mt_keys(1060, (1 << q) // 60)]), sync)
        apply(gqf, cuda, f, c, "delete", many, sync)
    finally:
        gqf.freeFilterGPU(f)


@pytest.mark.parametrize("sync", [True, False])
@pytest.mark.parametrize("op", ["insert", "delete", "merge", "via"])
@pytest.mark.parametrize("q,lo,width", [(16, 100, 2130), (7, 20, 3), (11, 500, 50), (12, 40, 120), (13, 300, 260)])
def test_dense_range(gqf, cuda, op, q, lo, width, sync):
    """Nearly every remainder of neighbouring quotients, in one cluster that no
    slice of the table holds: at q = 16 more items than a bucket of the rebuild
    counts in 16 bits, and filters smaller than one bucket."""
    G, r = gqf, 5
    cand = O.mt_keys(1130, 1 << (23 if q == 16 else 20))
    quot = O.aphash(cand, q, r) >> r
    dense = cand[(quot >= lo) & (quot < lo + width)]
    if q == 16:
        assert 66000 < np.unique(O.aphash(dense, q, r)).size < 68160
    more = O.mt_keys(1131, (1 << q) // 32)
    c = Contents(q, r, dense, True)
    f, f2 = G.initFilterGPU(q, r), G.initFilterGPU(q, r)
    try:
        G.bulkBuildSegmentedLayouts(f, dense.size, to_dev(cuda, dense), True)
        d = to_dev(cuda, more)
        if op == "insert":
            c.insert(more)
            G.insert(f, more.size, d, sync=sync)
        elif op == "delete":
            gone = np.concatenate([dense[: dense.size // 50], more])
            c.delete(gone)
            G.superclusterDeletes(f, gone.size, to_dev(cuda, gone), sync=sync)
        elif op == "via":
            c.merge(c.fps(more), True)
            G.insertViaMerge(f, d, 0, d, more.size, True, sync=sync)
        else:
            c.merge(np.unique(c.fps(more)), True)
            G.bulkBuildSegmentedLayouts(f2, more.size, d, True)
            G.mergeTwoFilters(f, f2, True, sync=sync)
        G.stream_status()
        check(G, f, c.table(), op)
    finally:
        G.freeFilterGPU(f)
        G.freeFilterGPU(f2)


@pytest.mark.parametrize("sync", [True, False])
@pytest.mark.parametrize("q", [9, 14, 17, 23])
def test_large_repeating_batches_on_a_table_with_copies(gqf, cuda, q, sync):
    """Batches of many times the table's buckets, mostly repeats: the rebuild
    keeps of them what changes the table."""
    r = 5
    n = min((1 << q) // 2, 1 << 20)
    cand = O.mt_keys(1140 + q, 2 * n)
    keys = np.concatenate([cand[:n], cand[: n // 4], np.repeat(cand[n: n + 3], 40 if q == 9 else 300)])
    hot = np.concatenate([np.full(90000, cand[n], np.uint32), np.full(70000, cand[n + 5], np.uint32), cand[: n // 8],
                          cand[-n // 8:], np.tile(cand[n // 3: n // 3 + 50], 200)])
    f, c = gqf.initFilterGPU(q, r), Contents(q, r, keys, False)
    assert c.table() is not None
    try:
        gqf.bulkBuildSegmentedLayouts(f, keys.size, to_dev(cuda, keys), False)
        apply(gqf, cuda, f, c, "insert", hot, sync)
        apply(gqf, cuda, f, c, "delete", hot, sync)
        apply(gqf, cuda, f, c, "delete", np.concatenate([hot[:100000], cand[: n // 2]]), sync)
    finally:
        gqf.freeFilterGPU(f)


@pytest.mark.parametrize("q,na,nb", [(7, 0.4, 0.4), (12, 0.5, 0.3), (16, 0.5, 0.5), (22, 0.5, 0.55), (23, 0.2, 0.2)])
@pytest.mark.parametrize("dup", [False, True])
def test_queued_merges(gqf, cuda, q, na, nb, dup):
    """Unique merges, of tables with copies too (which the in-place form
    unites as well), and a key batch merged in."""
    G, r = gqf, 5
    a, b = O.mt_keys(1070 + q, int(na * (1 << q))), O.mt_keys(1090 + q, int(nb * (1 << q)))
    c = O.mt_keys(1110 + q, (1 << q) // 32)
    if dup:
        a, b = np.concatenate([a[: a.size // 2]] * 2), np.concatenate([b, b[:9]])
    ca, cb = Contents(q, r, a, not dup), Contents(q, r, b, not dup)
    fa, fb = G.initFilterGPU(q, r), G.initFilterGPU(q, r)
    try:
        G.bulkBuildSegmentedLayouts(fa, a.size, to_dev(cuda, a), not dup)
        G.bulkBuildSegmentedLayouts(fb, b.size, to_dev(cuda, b), not dup)
        G.mergeTwoFilters(fa, fb, True, sync=False)
        G.insertViaMerge(fa, None, 0, to_dev(cuda, c), c.size, True, sync=False)
        G.stream_status()
        ca.merge(cb.f, True)
        ca.merge(ca.fps(c), True)
        check(G, fa, ca.table(), "first")
        check(G, fb, cb.table(), "second")  # only read
    finally:
        G.freeFilterGPU(fa)
        G.freeFilterGPU(fb)

"""SQF lookups on both sides of the rule that chooses between direct probes and
the bit-plane mirror, sorted and unsorted, queued and synchronous."""
import numpy as np
import pytest

import oracle as O
from conftest import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q,r,alpha,nodup", [(7, 5, 0.9, True), (13, 5, 1.02, True), (18, 5, 0.8, False),
                                             (12, 13, 1.03, True), (15, 13, 0.8, False)])
@pytest.mark.parametrize("n", [1, 4097, (3 << 18) - 1, 3 << 18])
def test_lookup_paths(gqf, cuda, q, r, alpha, nodup, n):
    keys = O.mt_keys(800 + q, int(alpha * (1 << q)))
    t = O.sqf_new(q, r)
    assert O.sqf_bulk_build(t, q, r, keys, nodup) == 0
    base = np.concatenate([keys, O.mt_keys(801 + q, keys.size)])
    base = base[np.random.default_rng(2).permutation(base.size)]
    reps = -(-n // base.size)
    look, want = np.tile(base, reps)[:n], np.tile(O.sqf_lookup(t, q, r, base), reps)[:n]
    f = gqf.initFilterGPU(q, r)
    try:
        gqf.bulkBuildSegmentedLayouts(f, keys.size, to_dev(cuda, keys), nodup)
        for op in (gqf.launchUnsortedLookups, gqf.launchSortedLookups):
            for sync in (True, False):
                out = cuda.zeros(n, dtype=cuda.int32, device="cuda")
                op(f, n, to_dev(cuda, look), out, sync=sync)
                gqf.stream_status()
                assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
    finally:
        gqf.freeFilterGPU(f)

"""RSQF lookups through the aligned mirror (batches of a million queries and
more, here the same ones over and over): the oracle's answers on regular and irregular tables (incremental
batches, spills over several blocks, a nearly full filter, the last blocks),
and the same as the direct lookups of small batches."""
import numpy as np
import pytest

import oracle as O
from conftest import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rbits", [5, 8])
@pytest.mark.parametrize("q,alpha,batches,hot", [(7, 0.9, 1, 0), (11, 0.6, 3, 0), (14, 0.95, 2, 0), (15, 0.4, 1, 600),
                                                 (16, 0.99, 1, 0)])
def test_mirror_lookups(gqf, cuda, q, alpha, batches, hot, rbits):
    n = int(alpha * (1 << q))
    keys = O.mt_keys(600 + q, n)
    if hot:  # many items in a narrow quotient range: offsets of several blocks
        cand = O.mt_keys(601, 1 << 19)
        keys = np.concatenate([keys, cand[(O.aphash(cand, q, rbits) >> rbits) < hot // 2][:hot]])
    f = gqf.initCQFGPU(q, rbits)
    try:
        parts = np.array_split(keys, batches + 1)  # the first build, then incremental batches
        for p in parts:
            ret = cuda.empty(max(p.size, 1), dtype=cuda.int32, device="cuda")
            gqf.insertGPU(f, p.size, to_dev(cuda, p), ret)
        o = O.rsqf_new(q, rbits)
        for p in parts:
            O.rsqf_insert_sorted(o, q, p, rbits)
        assert np.array_equal(gqf.rsqf_blocks_bytes(f), o)
        look = np.concatenate([keys, O.mt_keys(602 + q, max(keys.size, 64))])
        want = O.rsqf_lookup(o, q, look, rbits)
        reps = -(-(3 << 19) // look.size)
        look, want = np.tile(look, reps), np.tile(want, reps)
        for op in (gqf.launchLookups, gqf.launchUnsortedLookupsRSQF):
            out = cuda.empty(look.size, dtype=cuda.int32, device="cuda")
            op(f, look.size, to_dev(cuda, look), out)
            assert np.array_equal(out.cpu().numpy(), want)
            m = max(1, (1 << q) // 32)
            out = cuda.empty(m, dtype=cuda.int32, device="cuda")
            op(f, m, to_dev(cuda, look[-m:].copy()), out)
            assert np.array_equal(out.cpu().numpy(), want[-m:])
    finally:
        gqf.freeCQFGPU(f)

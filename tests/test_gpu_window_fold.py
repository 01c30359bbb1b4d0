"""Results of records cut into one to thousands of windows, where the same score
comes back in many of them, against the oracle: the first row and the smallest
column win."""
import numpy as np
import pytest

import oracle as O
from ish_gb300 import native
from ish_gb300.scoring import ScoringMatrix
from test_gpu_parity import THREADS, ctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 200])
@pytest.mark.parametrize("algo, ends", [(native.ALGO_SEMI_GLOBAL, 12), (native.ALGO_SEMI_GLOBAL, 13), (native.ALGO_LOCAL, 0)])
def test_ties_between_windows(ctx, algo, ends, n):  # noqa: F811
    rng = np.random.default_rng(n)
    q = rng.integers(0, 4, 18, dtype=np.uint8)
    lens = rng.integers(0, 60, n)
    lens[rng.permutation(n)[:5]] = [700_000, 9_000, 8_700, 30_001, 500][:min(n, 5)]
    off = np.concatenate(([0], np.cumsum(lens))).astype(np.uint64)
    buf = rng.integers(0, 4, int(off[-1]), dtype=np.uint8)
    for i in range(n):  # the query every 97 rows: equal maxima in all windows of most records
        for at in range(int(off[i]) + int(rng.integers(0, 60)), int(off[i + 1]) - 18, 97):
            if i % 3:
                buf[at:at + 18] = q
    m = ScoringMatrix(O.ACTGN)
    best = int(m.values[q, q].astype(np.int64).sum())
    qid = ctx.set_query(q, O.ACTGN, m.values, algo, 3, 1, ends, best, 0.6)
    om = O.Matcher(O.SEMI_GLOBAL if algo == native.ALGO_SEMI_GLOBAL else O.LOCAL, O.ACTGN, q, best, 0.6,
                   gap_open=3, gap_extend=1, ends=ends)
    sid = ctx.records_load(buf, off)
    g = ctx.score_set(qid, sid)
    assert ctx.last_windows() > 1000
    o = om.batch(buf, off, threads=THREADS)
    for k in ("score", "qend", "tend", "hit"):
        assert (g[k] == o[k]).all(), k
    ctx.records_free(sid)
    ctx.free_query(qid)

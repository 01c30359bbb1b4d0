"""Queries that come and go: each one's first launch reads its own profile and not
what the same memory held for the query before, against the oracle."""
import numpy as np
import pytest

import oracle as O
from ish_gb300 import native
from ish_gb300.scoring import ScoringMatrix
from test_gpu_parity import THREADS, ctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", [native.ALGO_SEMI_GLOBAL, native.ALGO_LOCAL])
@pytest.mark.parametrize("qlen", [2, 24, 120])
def test_first_launches(ctx, algo, qlen):  # noqa: F811
    rng = np.random.default_rng(qlen + algo)
    m = ScoringMatrix(O.ACTGN)
    lens = rng.integers(0, 60, 150)
    off = np.concatenate(([0], np.cumsum(lens))).astype(np.uint64)
    buf = rng.integers(0, 4, int(off[-1]), dtype=np.uint8)
    sid = ctx.records_load(buf, off)
    queries = [rng.integers(0, 4, qlen, dtype=np.uint8) for _ in range(5)]
    best = [int(m.values[q, q].astype(np.int64).sum()) for q in queries]
    want = [O.Matcher(O.SEMI_GLOBAL if algo == native.ALGO_SEMI_GLOBAL else O.LOCAL, O.ACTGN, q, b, 0.6, gap_open=3,
                      gap_extend=1, ends=12).batch(buf, off, threads=THREADS) for q, b in zip(queries, best)]
    for turn in range(400):
        i = turn % 5
        qid = ctx.set_query(queries[i], O.ACTGN, m.values, algo, 3, 1, 12, best[i], 0.6)
        g = ctx.score(qid, buf, off) if turn & 1 else ctx.score_set(qid, sid)
        for k in ("score", "qend", "tend", "hit"):
            assert (g[k] == want[i][k]).all(), (turn, k)
        ctx.free_query(qid)
    ctx.records_free(sid)

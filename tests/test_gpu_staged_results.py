"""Results of small calls written straight to pinned memory: every choice of
outputs, at the edges of the staging area, against the oracle."""
import numpy as np
import pytest

from ish_gb300 import native
from test_gpu_parity import THREADS, ctx  # noqa: F401
from test_gpu_small_sets import make_query, random_set

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 5, 4095, 4096, 4097])
def test_choices_of_outputs(ctx, n):  # noqa: F811
    rng = np.random.default_rng(n)
    buf, off = random_set(rng, n, 300)
    qid, om = make_query(ctx, rng.integers(0, 4, 5, dtype=np.uint8), native.ALGO_SEMI_GLOBAL)
    o = om.batch(buf, off, threads=THREADS)
    o["hit_idx"] = np.nonzero(o["hit"])[0].astype(np.uint32)
    sid = ctx.records_load(buf, off)
    for want in (("score",), ("hit_idx",), ("hit", "hit_idx"), ("qend", "tend"),
                 ("score", "qend", "tend", "hit", "hit_idx")):
        for g in (ctx.score(qid, buf, off, want=want), ctx.score_set(qid, sid, want=want)):
            for k in want:
                assert (g[k] == o[k]).all() and len(g[k]) == len(o[k]), (n, want, k)
    ctx.records_free(sid)
    ctx.free_query(qid)

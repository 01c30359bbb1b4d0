"""Starts of hits that end past the lengths a set's histogram tells apart,
against the oracle's starts."""
import numpy as np
import pytest

from ish_gb300 import native
from test_gpu_parity import ctx  # noqa: F401
from test_gpu_small_sets import make_query

pytestmark = pytest.mark.gpu
LAST_BUCKET = 32768 + 32767 * 32  # lengths from here on share a bucket


@pytest.mark.parametrize("algo", [native.ALGO_SEMI_GLOBAL, native.ALGO_LOCAL])
@pytest.mark.parametrize("n", [5, 4200])
def test_hits_at_the_end_of_long_records(ctx, algo, n):  # noqa: F811
    rng = np.random.default_rng(n + algo)
    q = rng.integers(0, 4, 24, dtype=np.uint8)
    lens = rng.integers(0, 60, n)
    long = {0: LAST_BUCKET + 31, 2: LAST_BUCKET + 32, 3: 1_200_007, n - 1: 2_000_000}
    for i, length in long.items():
        lens[i] = length
    off = np.concatenate(([0], np.cumsum(lens))).astype(np.uint64)
    buf = rng.integers(0, 4, int(off[-1]), dtype=np.uint8)
    for i in long:
        buf[int(off[i + 1]) - 24:int(off[i + 1])] = q
    qid, om = make_query(ctx, q, algo)
    sid = ctx.records_load(buf, off)
    tend = ctx.score_set(qid, sid)["tend"]
    h = np.array(list(long) * 3, np.uint32)
    starts = ctx.match_starts(qid, sid, h, tend[h])
    for i, start in zip(h, starts):
        assert tend[i] == lens[i] - 1
        assert start == om.first_match(buf[int(off[i]):int(off[i + 1])])[0] == lens[i] - 24, (i, lens[i])
    ctx.records_free(sid)
    ctx.free_query(qid)

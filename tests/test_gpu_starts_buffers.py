"""Start finding with buffers kept between calls: hit counts around the staging
area, ends outside their records, and sets that take a freed set's buffers,
against the oracle's starts."""
import numpy as np
import pytest

import oracle as O
from ish_gb300 import native
from test_gpu_parity import ctx  # noqa: F401
from test_gpu_small_sets import make_query, random_set

pytestmark = pytest.mark.gpu


def hits_of(n, rng, count):
    return rng.integers(0, n, count).astype(np.uint32)  # repeats, any order


@pytest.mark.parametrize("algo", [native.ALGO_SEMI_GLOBAL, native.ALGO_LOCAL])
def test_counts_and_ends(ctx, algo):  # noqa: F811
    rng = np.random.default_rng(5 + algo)
    q = rng.integers(0, 4, 20, dtype=np.uint8)
    qid, om = make_query(ctx, q, algo)
    for n in (3000, 200, 5000):  # each set takes the freed one's buffers
        buf, off = random_set(rng, n, 700)
        lens = np.diff(off).astype(np.int64)
        sid = ctx.records_load(buf, off)
        s = ctx.score_set(qid, sid)
        one = ctx.match_starts(qid, sid, np.arange(n, dtype=np.uint32), s["tend"])
        for i in range(0, n, 97):
            if s["hit"][i]:
                assert one[i] == om.first_match(buf[int(off[i]):int(off[i + 1])])[0], (n, i)
        for count in (1, 3, 8703, 8704, 8705, 20000):
            h = hits_of(n, rng, count)
            assert (ctx.match_starts(qid, sid, h, s["tend"][h]) == one[h]).all(), (n, count)
        h = hits_of(n, rng, 500)
        last = ctx.match_starts(qid, sid, h, (lens[h] - 1).astype(np.int32))
        for past in (0, 5, 1 << 30):  # an end past its record counts as its last residue
            ends = np.minimum(lens[h] - 1 + past, 2**31 - 1).astype(np.int32)
            assert (ctx.match_starts(qid, sid, h, ends) == last).all(), (n, past)
        assert (ctx.match_starts(qid, sid, h, np.full(500, -1, np.int32)) == -1).all()
        ctx.records_free(sid)
    ctx.free_query(qid)

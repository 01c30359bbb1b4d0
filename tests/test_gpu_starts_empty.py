"""Starts of empty prefixes next to ones long enough to be cut into windows."""
import numpy as np
import pytest

from ish_gb300 import native
from test_gpu_parity import ctx  # noqa: F401
from test_gpu_small_sets import make_query, random_set

pytestmark = pytest.mark.gpu


def test_empty_prefixes_in_a_windowed_pass(ctx):  # noqa: F811
    rng = np.random.default_rng(6)
    q = rng.integers(0, 4, 20, dtype=np.uint8)
    qid, _ = make_query(ctx, q, native.ALGO_LOCAL)
    buf, off = random_set(rng, 200, 2000)
    end = int(off[np.argmax(np.diff(off)) + 1])
    buf[end - 20:end] = q  # the long record's end: its prefix is cut into windows
    sid = ctx.records_load(buf, off)
    tend = ctx.score_set(qid, sid)["tend"]
    h = rng.integers(0, 200, 8703).astype(np.uint32)
    one = np.concatenate([ctx.match_starts(qid, sid, h[i:i + 1], tend[h[i:i + 1]]) for i in range(0, 8703, 50)])
    many = ctx.match_starts(qid, sid, h, tend[h])
    assert ctx.last_windows() > 8703  # more windows than prefixes
    assert (many[::50] == one).all() and (many[tend[h] < 0] == -1).all()
    ctx.records_free(sid)
    ctx.free_query(qid)

"""Batched and served searches of records whose lengths share the sort's last bucket,
the first of them not the longest, against the oracle."""
import numpy as np
import pytest

import oracle as O
from ish_gb300 import native
from ish_gb300.scoring import ScoringMatrix
from test_gpu_parity import THREADS, ctx  # noqa: F401

pytestmark = pytest.mark.gpu
LAST_BUCKET = 32768 + 32767 * 32


@pytest.mark.parametrize("ends", [15, 12])
@pytest.mark.parametrize("lens", [[LAST_BUCKET - 1], [LAST_BUCKET, LAST_BUCKET + 40], [LAST_BUCKET + 1, 2_000_000],
                                  [50, LAST_BUCKET + 5, 30, 1_600_001, 1_300_000]])
def test_longest_record_last(ctx, ends, lens):  # noqa: F811
    rng = np.random.default_rng(len(lens))
    m = ScoringMatrix(O.ACTGN)
    off = np.concatenate(([0], np.cumsum(lens))).astype(np.uint64)
    buf = rng.integers(0, 4, int(off[-1]), dtype=np.uint8)
    sid = ctx.records_load(buf, off)
    qids, want = [], []
    for Q in (20, 45):
        q = rng.integers(0, 4, Q, dtype=np.uint8)
        best = int(m.values[q, q].astype(np.int64).sum())
        qids.append(ctx.set_query(q, O.ACTGN, m.values, native.ALGO_SEMI_GLOBAL, 3, 1, ends, best, 0.4))
        want.append(O.Matcher(O.SEMI_GLOBAL, O.ACTGN, q, best, 0.4, gap_open=3, gap_extend=1, ends=ends).batch(
            buf, off, threads=THREADS))
    r = ctx.score_multi(qids, sid)
    for i, o in enumerate(want):
        for k in ("score", "qend", "tend", "hit"):
            assert (r[k][i] == o[k]).all(), (i, k)
    ctx.serve_start(sid)
    try:
        for t, o in [(ctx.submit(q), o) for q, o in zip(qids, want)]:
            g = None
            while g is None:
                g = ctx.poll(t, 200)
            assert np.array_equal(g["hit_idx"], np.nonzero(o["hit"])[0])
    finally:
        ctx.serve_stop()
    for q in qids:
        ctx.free_query(q)
    ctx.records_free(sid)

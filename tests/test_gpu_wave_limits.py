"""Wavefront scoring where its 16-bit values and its record ends can go wrong:
the deepest boundaries and the largest penalties that the fast regime admits,
and pairs of records that end in every row of a pipeline step, against the
oracle, bit for bit."""
import numpy as np
import pytest

import oracle as O
from ish_gb300 import native
from test_gpu_parity import ALL_ENDS, assert_same, ctx, run_both  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qlen,gap_open,gap_ext,longest", [
    (2040, 9, 1, 25000),   # the widest query and the longest record of a fixed target start
    (50, 9990, 9, 900),    # the dearest opening
    (40, 520, 510, 40),    # frames that reset every four rows
    (300, 600, 2, 12000),
])
def test_semi_global_value_range(ctx, qlen, gap_open, gap_ext, longest):  # noqa: F811
    rng = np.random.default_rng(qlen + gap_ext)
    q = rng.integers(0, 20, qlen, dtype=np.uint8)
    recs = [rng.integers(0, 20, int(n), dtype=np.uint8) for n in rng.integers(1, 2 * qlen, 10)]
    recs += [np.tile(q, 3)[:longest], rng.integers(0, 20, longest, dtype=np.uint8),
             np.full(min(longest, 4000), 17, np.uint8)]
    for ends in ALL_ENDS:
        g, o = run_both(ctx, native.ALGO_SEMI_GLOBAL, O.BLOSUM62, q, recs, gap_open, gap_ext, ends, thr=0.1)
        assert_same(g, o, f"Q={qlen} gaps={gap_open}/{gap_ext} ends={ends}")


@pytest.mark.parametrize("G,qlen", [(1, 1), (1, 24), (2, 24), (4, 9), (8, 100), (32, 40)])
@pytest.mark.parametrize("algo", [native.ALGO_SEMI_GLOBAL, native.ALGO_LOCAL])
def test_record_ends_in_every_row_of_a_step(ctx, algo, G, qlen):  # noqa: F811
    rng = np.random.default_rng(G + qlen)
    q = rng.integers(0, 4, qlen, dtype=np.uint8)
    recs = [rng.integers(0, 4, n, dtype=np.uint8) for n in list(range(0, 71)) * 3 + [140, 3, 129, 64]]
    try:
        ctx.set_option(native.OPT_WAVE_GROUP, G)
        for ends in ALL_ENDS if algo == native.ALGO_SEMI_GLOBAL else (0,):
            g, o = run_both(ctx, algo, O.ACTGN, q, recs, 3, 1, ends, thr=0.3)
            assert_same(g, o, f"G={G} Q={qlen} ends={ends}")
    finally:
        ctx.set_option(native.OPT_WAVE_GROUP, 0)

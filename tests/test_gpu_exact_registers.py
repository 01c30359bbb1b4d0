"""The lane-exact passes with their stripes in registers: every stripe count
they are compiled for and the one past it, tiles of a warp that end at
different rows, saturating records, against the oracle for the same lanes."""
import numpy as np
import pytest

import oracle as O
from ish_gb300 import native
from test_gpu_exact import both, ctx, recs_with_copies  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [8, 16, 32])
@pytest.mark.parametrize("segs", [1, 2, 3, 4, 5, 6, 7, 8, 9, 12, 13, 16, 17, 24, 25, 32, 33])
def test_stripe_counts(ctx, lanes, segs):  # noqa: F811
    rng = np.random.default_rng(100 * lanes + segs)
    for qlen in {lanes * segs, lanes * (segs - 1) + 1}:
        if qlen > 300:
            continue
        q = rng.integers(0, 20, qlen, dtype=np.uint8)
        # 0 to 3 records past a warp's tiles, of any length down to none
        recs = recs_with_copies(rng, 20, q, 61 + segs % 4, 0, qlen + 90, frac=0.5, sub=0.05)
        recs += [np.zeros(0, np.uint8), np.tile(q, 2), rng.integers(0, 20, 700, dtype=np.uint8)]
        for gaps in ((2, 2), (1, 3), (0, 0)):
            for ends in (0, 7, 12, 15):
                both(ctx, native.ALGO_SEMI_GLOBAL, O.BLOSUM62, q, recs, *gaps, ends, lanes=(lanes, 16, 8))
            both(ctx, native.ALGO_LOCAL, O.BLOSUM62, q, recs, *gaps, 0, lanes=(8, lanes, lanes))


def test_one_record_and_boundaries_that_wrap(ctx):  # noqa: F811
    rng = np.random.default_rng(9)
    for qlen in (30, 120, 250):
        q = rng.integers(0, 20, qlen, dtype=np.uint8)
        for recs in ([q], [rng.integers(0, 20, n, dtype=np.uint8) for n in (34000, 33000, 70000, 90, 4)]):
            for ends in (0, 3, 8, 11, 12):
                both(ctx, native.ALGO_SEMI_GLOBAL, O.BLOSUM62, q, recs, 1, 1, ends)
            both(ctx, native.ALGO_LOCAL, O.BLOSUM62, q, recs, 1, 1, 0)

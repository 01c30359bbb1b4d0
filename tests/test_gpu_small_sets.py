"""Sets that one block sorts and packs, and hits that one block compacts, at
the edges of both, against the oracle."""
import numpy as np
import pytest

import oracle as O
from ish_gb300 import native
from ish_gb300.scoring import ScoringMatrix
from test_gpu_parity import THREADS, assert_same, ctx  # noqa: F401

pytestmark = pytest.mark.gpu


def random_set(rng, n, longest):
    lens = rng.integers(0, 40, n)
    lens[rng.random(n) < 0.1] = 0
    lens[rng.integers(n)] = longest
    off = np.concatenate(([0], np.cumsum(lens))).astype(np.uint64)
    return rng.integers(0, 4, int(off[-1]), dtype=np.uint8), off


def make_query(ctx, q, algo):  # noqa: F811
    m = ScoringMatrix(O.ACTGN)
    best = int(m.values[q, q].astype(np.int64).sum())
    om = O.Matcher(O.SEMI_GLOBAL if algo == native.ALGO_SEMI_GLOBAL else O.LOCAL, O.ACTGN, q, best, 0.6,
                   gap_open=3, gap_extend=1, ends=15)
    return ctx.set_query(q, O.ACTGN, m.values, algo, 3, 1, 15, best, 0.6), om


@pytest.mark.parametrize("n", [1, 2, 3, 1023, 1024, 1025, 4095, 4096, 4097])
def test_small_sets(ctx, n):  # noqa: F811
    rng = np.random.default_rng(n)
    buf, off = random_set(rng, n, 33003)
    shifted = np.concatenate((np.full(13, 3, np.uint8), buf))  # the first record may start anywhere
    q = rng.integers(0, 4, 12, dtype=np.uint8)
    for algo in (native.ALGO_SEMI_GLOBAL, native.ALGO_LOCAL):
        qid, om = make_query(ctx, q, algo)
        o = om.batch(buf, off, threads=THREADS)
        assert_same(ctx.score(qid, buf, off), o, f"n={n}")
        assert_same(ctx.score(qid, shifted, off + np.uint64(13)), o, f"n={n} from 13")
        for load in (ctx.records_load, ctx.records_load_async):
            sid = load(shifted, off + np.uint64(13))
            assert_same(ctx.score_set(qid, sid), o, f"n={n} {load.__name__}")
            codes, offsets = ctx.records_get(sid)
            assert (codes == buf).all() and (offsets == off).all()
            ctx.records_free(sid)
        ctx.free_query(qid)


@pytest.mark.parametrize("n", [1, 500, 4096, 4097])
def test_codes_outside_the_alphabet(ctx, n):  # noqa: F811
    rng = np.random.default_rng(n)
    buf, off = random_set(rng, n, 200)
    q = rng.integers(0, 4, 12, dtype=np.uint8)
    for algo in (native.ALGO_SEMI_GLOBAL, native.ALGO_LOCAL):
        qid, om = make_query(ctx, q, algo)
        for code in (ScoringMatrix(O.ACTGN).size, 255):
            bad = buf.copy()
            bad[rng.integers(len(bad))] = code
            for want in (("score", "qend", "tend", "hit", "hit_idx"), ("score",)):
                with pytest.raises(native.IshGpuError, match=f"code {code} >= the alphabet"):
                    ctx.score(qid, bad, off, want=want)
        assert_same(ctx.score(qid, buf, off), om.batch(buf, off, threads=THREADS), f"n={n}")
        ctx.free_query(qid)


@pytest.mark.parametrize("n", [16383, 16384, 16385, 40000])
def test_compaction(ctx, n):  # noqa: F811
    rng = np.random.default_rng(n)
    q = rng.integers(0, 4, 8, dtype=np.uint8)
    lens = rng.integers(4, 14, n)
    off = np.concatenate(([0], np.cumsum(lens))).astype(np.uint64)
    buf = rng.integers(0, 4, int(off[-1]), dtype=np.uint8)
    qid, om = make_query(ctx, q, native.ALGO_SEMI_GLOBAL)
    o = om.batch(buf, off, threads=THREADS)
    assert 0 < o["hit"].sum() < n
    assert_same(ctx.score(qid, buf, off), o, f"n={n}")
    ctx.free_query(qid)

"""After the autotuner has timed a query's shapes, a set with few records still gets
one of its own, on a runtime without a device (where all times are equal)."""
import pytest

from fake_device import fake_lib, run  # noqa: F401


@pytest.mark.parametrize("mode, Q", [(0, 120), (1, 120), (0, 463), (1, 800)])
def test_small_set_keeps_its_shape(fake_lib, mode, Q):  # noqa: F811
    run(fake_lib, f"""
from ish_gb300.scoring import BLOSUM62, ScoringMatrix
m = ScoringMatrix(BLOSUM62)
rng = np.random.default_rng(3000)
lens = np.clip(rng.lognormal(np.log(320), 0.6, 3000), 30, 8000).astype(int)
off = np.concatenate(([0], np.cumsum(lens))).astype(np.uint64)
sid = ctx.records_load(np.zeros(int(off[-1]), np.uint8), off)
ctx.set_option(native.OPT_WINDOWS, 0)
q = np.random.default_rng({Q}).integers(0, 20, {Q}, dtype=np.uint8)
qid = ctx.set_query(q, BLOSUM62, m.values, {mode}, 10, 1, 12, 1000, 0.5)
ctx.score_set(qid, sid)
before = last_wave()
group, cols = ctx.autotune(sid, [qid])
ctx.score_set(qid, sid)
assert last_wave() == before and before[0] < cols[0], (before, group, cols, last_wave())
""")

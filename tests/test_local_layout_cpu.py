"""Profile layouts of long local queries: 32-bit words only where all of an SM's
threads fit beside them, on a runtime without a device."""
import pytest

from fake_device import fake_lib, run  # noqa: F401

S32, S16 = 2, 0


@pytest.mark.parametrize("Q, layout", [(300, S32), (1663, S32), (1727, S16), (1791, S16), (1919, S16), (2047, S16)])
def test_layout(fake_lib, Q, layout):  # noqa: F811
    run(fake_lib, f"""
from ish_gb300.scoring import BLOSUM62, ScoringMatrix
m = ScoringMatrix(BLOSUM62)
off = np.arange(4001, dtype=np.uint64) * 350
sid = ctx.records_load(np.zeros(int(off[-1]), np.uint8), off)
q = np.random.default_rng(1).integers(0, 20, {Q}, dtype=np.uint8)
qid = ctx.set_query(q, BLOSUM62, m.values, native.ALGO_LOCAL, 10, 1, 0, 1000, 0.5)
ctx.score_set(qid, sid)
assert last_wave()[1:3] == (1, {layout}), last_wave()
""")

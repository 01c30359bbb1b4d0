"""Profile layouts of queries with a free query end: the copies of the last row
stay in L1 beside the profile, on a runtime without a device."""
import pytest

from fake_device import fake_lib, run  # noqa: F401

PAIR, S32, S16 = 1, 2, 0


@pytest.mark.parametrize("residues, Q, ends, layout", [
    (4, 1407, 15, PAIR), (4, 1535, 15, S32), (4, 2047, 15, S32), (4, 2047, 13, PAIR),
    (20, 1663, 15, S32), (20, 1983, 15, S16), (20, 2047, 15, S16), (20, 2047, 13, S32), (20, 300, 15, S32)])
def test_layout(fake_lib, residues, Q, ends, layout):  # noqa: F811
    run(fake_lib, f"""
from ish_gb300.scoring import BLOSUM62, ScoringMatrix
kind = 1 if {residues} == 4 else BLOSUM62
m = ScoringMatrix(kind)
off = np.arange(1001, dtype=np.uint64) * 150
sid = ctx.records_load(np.zeros(int(off[-1]), np.uint8), off)
q = np.random.default_rng(1).integers(0, {residues}, {Q}, dtype=np.uint8)
qid = ctx.set_query(q, kind, m.values, native.ALGO_SEMI_GLOBAL, 10, 1, {ends}, 1000, 0.5)
ctx.score_set(qid, sid)
assert last_wave()[1:3] == (0, {layout}), last_wave()
""")

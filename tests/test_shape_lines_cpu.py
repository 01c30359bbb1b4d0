"""Shapes that queries get for sets of short lines, against those that were the
fastest of all when each was timed, on a runtime without a device."""
import pytest

from fake_device import fake_lib, run  # noqa: F401


# lines, mode, bytes of the query: columns per thread within 6 % of the fastest
@pytest.mark.parametrize("lines, cases", [
    (500, [(0, 24, {4, 7}), (0, 60, {8}), (1, 60, {8})]),
    (100_000, [(0, 24, {13, 25}), (0, 40, {21, 42}), (0, 60, {16})]),
    (300_000, [(0, 24, {25}), (0, 40, {21, 42}), (0, 60, {16}), (1, 24, {25})])])
def test_shapes(fake_lib, lines, cases):  # noqa: F811
    run(fake_lib, f"""
from ish_gb300.scoring import ScoringMatrix
m = ScoringMatrix(0)
lens = np.random.default_rng({lines}).integers(20, 121, {lines})
off = np.concatenate(([0], np.cumsum(lens))).astype(np.uint64)
sid = ctx.records_load(np.zeros(int(off[-1]), np.uint8), off)
for mode, Q, columns in {cases!r}:
    q = np.random.default_rng(Q).integers(0x20, 0x7f, Q, dtype=np.uint8)
    qid = ctx.set_query(q, 0, m.values, mode, 3, 1, 12, 100, 0.8)
    ctx.score_set(qid, sid)
    assert last_wave()[0] in columns and last_wave()[1] == mode, (mode, Q, last_wave())
    ctx.free_query(qid)
""")

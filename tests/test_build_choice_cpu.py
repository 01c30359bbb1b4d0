"""Builds of wide local rows by profile layout, against the faster one when both
were timed, on a runtime without a device."""
import pytest

from fake_device import fake_lib, run  # noqa: F401


@pytest.mark.parametrize("kind, residues, lean", [(1, 4, {34: 0, 42: 0, 44: 0, 48: 0, 29: 1}),
                                                  (3, 20, {34: 0, 38: 0, 44: 1, 46: 1, 48: 1, 29: 1})])
def test_builds(fake_lib, kind, residues, lean):  # noqa: F811
    run(fake_lib, f"""
from ish_gb300.scoring import ScoringMatrix
m = ScoringMatrix({kind})
off = np.arange(200001, dtype=np.uint64) * 150
sid = ctx.records_load(np.zeros(int(off[-1]), np.uint8), off)
ctx.set_option(native.OPT_WAVE_GROUP, 8)
for K, lean in {lean!r}.items():
    ctx.set_option(native.OPT_WAVE_K, K)
    q = np.random.default_rng(K).integers(0, {residues}, 8 * K - 2, dtype=np.uint8)
    qid = ctx.set_query(q, {kind}, m.values, native.ALGO_LOCAL, 10, 1, 0, 1000, 0.5)
    ctx.score_set(qid, sid)
    assert last_wave() == (K, 1, {1 if kind == 1 else 2}, lean), last_wave()
""")

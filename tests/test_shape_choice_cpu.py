"""Shapes and builds that queries get for a set of proteins, against those that
were the fastest of all when each was timed, on a runtime without a device."""
import pytest

from fake_device import fake_lib, run  # noqa: F401

# records, mode, residues: columns per thread that were within 5 % of the fastest,
# and the build (0 usual, 1 lean; None where the columns have one build or either
# will do)
CASES = [
    (3000, 0, 1000, {32}, 1), (3000, 1, 800, {26}, 1),
    (15000, 0, 1000, {32}, 1), (15000, 0, 1500, {48}, 1), (15000, 1, 1200, {38}, 1), (15000, 1, 800, {26}, 1),
    (60000, 0, 399, {25, 13}, None), (60000, 0, 463, {29, 15}, None), (60000, 0, 510, {32}, None),
    (60000, 1, 399, {25, 13}, None), (60000, 1, 430, {27, 14}, None), (60000, 1, 463, {29, 15}, None),
    (60000, 1, 1000, {32}, 1),
    (200000, 0, 214, {27}, None), (200000, 1, 1000, {32}, 1),
]


@pytest.mark.parametrize("records", sorted({c[0] for c in CASES}))
def test_shapes(fake_lib, records):  # noqa: F811
    cases = [c[1:] for c in CASES if c[0] == records]
    run(fake_lib, f"""
from ish_gb300.scoring import BLOSUM62, ScoringMatrix
m = ScoringMatrix(BLOSUM62)
rng = np.random.default_rng({records})
lens = np.clip(rng.lognormal(np.log(320), 0.6, {records}), 30, 8000).astype(int)
off = np.concatenate(([0], np.cumsum(lens))).astype(np.uint64)
sid = ctx.records_load(np.zeros(int(off[-1]), np.uint8), off)
ctx.set_option(native.OPT_WINDOWS, 0)
for mode, Q, columns, lean in {cases!r}:
    q = np.random.default_rng(Q).integers(0, 20, Q, dtype=np.uint8)
    qid = ctx.set_query(q, BLOSUM62, m.values, mode, 10, 1, 12, 1000, 0.5)
    ctx.score_set(qid, sid)
    got = last_wave()
    assert got[0] in columns and got[1] == mode and lean in (None, got[3]), (mode, Q, got)
    ctx.free_query(qid)
""")

"""Room for the reversed prefixes of hits in records longer than the last
bucket of a set's length histogram tells apart, on a runtime without a device."""
import pytest

from fake_device import fake_lib, run  # noqa: F401

LAST_BUCKET = 32768 + 32767 * 32  # lengths from here on share a bucket


@pytest.mark.parametrize("longest", [32767, LAST_BUCKET - 1, LAST_BUCKET + 31, LAST_BUCKET + 32, 2_000_000])
def test_prefixes_fit(fake_lib, longest):  # noqa: F811
    out = run(fake_lib, f"""
lens = np.array([40, {longest}, 0, 700])
off = np.concatenate(([0], np.cumsum(lens))).astype(np.uint64)
sid = ctx.records_load(np.zeros(int(off[-1]), np.uint8), off)
qid = ctx.set_query(np.zeros(20, np.uint8), 1, -np.ones((5, 5)) + 3 * np.eye(5), native.ALGO_LOCAL, 3, 1, 15, 40, 0.5)
ctx.score_set(qid, sid)
for ends in ([39, {longest} - 1, -1, 699], [2**31 - 1] * 4):
    for count in (4, 40):
        ctx.match_starts(qid, sid, np.arange(count) % 4, np.array(ends * 10)[:count])
print(fake.fake_report().decode())
""")
    assert "reversed prefixes" not in out

"""The arrays of a window view are uploaded before they are freed: single calls,
start finding and the serving thread, on a runtime without a device."""
import pytest

from fake_device import fake_lib, run  # noqa: F401


@pytest.mark.parametrize("n", [2, 300])
def test_uploads_end_before_their_sources(fake_lib, n):  # noqa: F811
    out = run(fake_lib, f"""
lens = np.full({n}, 40)
lens[0] = 60000
off = np.concatenate(([0], np.cumsum(lens))).astype(np.uint64)
sid = ctx.records_load(np.zeros(int(off[-1]), np.uint8), off)
qid = ctx.set_query(np.zeros(20, np.uint8), 1, -np.ones((5, 5)) + 3 * np.eye(5), native.ALGO_LOCAL, 3, 1, 15, 40, 0.5)
ctx.score_set(qid, sid)
assert ctx.last_windows() > {n}
ctx.match_starts(qid, sid, [0, 1], [59999, 39])
ctx.serve_start(sid)
ticket = ctx.submit(qid)
while ctx.poll(ticket, 100) is None:
    pass
ctx.serve_stop()
print(fake.fake_report().decode())
""")
    assert out.strip() == ""

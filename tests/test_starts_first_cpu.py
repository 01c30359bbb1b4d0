"""Start finding on a context that has not scored a set by itself before, on a
runtime without a device."""
from fake_device import fake_lib, run  # noqa: F401


def test_starts_are_the_first_launch(fake_lib):  # noqa: F811
    run(fake_lib, """
off = np.arange(51, dtype=np.uint64) * 300
sid = ctx.records_load(np.zeros(int(off[-1]), np.uint8), off)
qid = ctx.set_query(np.zeros(20, np.uint8), 1, -np.ones((5, 5)) + 3 * np.eye(5), native.ALGO_LOCAL, 3, 1, 15, 40, 0.5)
ctx.match_starts(qid, sid, np.arange(50), np.full(50, 299))
""")

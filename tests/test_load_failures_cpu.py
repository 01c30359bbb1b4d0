"""A load that fails part-way leaves no copy that still reads the caller's
buffers, on a runtime without a device."""
import pytest

from fake_device import fake_lib, run  # noqa: F401


@pytest.mark.parametrize("n", [3, 4096, 4097])
@pytest.mark.parametrize("copies", [0, 1, 2])
def test_no_copy_is_left_behind(fake_lib, n, copies):  # noqa: F811
    run(fake_lib, f"""
off = np.arange({n} + 1, dtype=np.uint64) * 30
buf = np.zeros(int(off[-1]), np.uint8)
qid = ctx.set_query(np.zeros(20, np.uint8), 1, -np.ones((5, 5)) + 3 * np.eye(5), native.ALGO_LOCAL, 3, 1, 15, 40, 0.5)
for load in (ctx.records_load, ctx.records_load_async, lambda b, o: ctx.score(qid, b, o)):
    fake.fake_refuse_copy_after({copies})
    try:
        load(buf, off)
    except native.IshGpuError:
        assert fake.fake_unread_uploads() == 0
    else:
        assert {copies} == 2, "the load makes more copies than were let through"
    fake.fake_refuse_copy_after(-1)
""")

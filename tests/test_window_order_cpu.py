"""Windows of a view go to the device longest first: in one group where one launch
scores them, by their place in the record where two do, on a runtime without a
device."""
import pytest

from fake_device import fake_lib, run  # noqa: F401


@pytest.mark.parametrize("mode, ends, split", [(1, 0, False), (0, 12, False), (0, 13, True)])
def test_longest_first(fake_lib, mode, ends, split):  # noqa: F811
    run(fake_lib, f"""
lens = np.random.default_rng(2).integers(20, 300, 400)
lens[:9] = [70000, 65000, 300, 40000, 30001, 9, 25000, 20000, 16000]
off = np.concatenate(([0], np.cumsum(lens))).astype(np.uint64)
sid = ctx.records_load(np.zeros(int(off[-1]), np.uint8), off)
qid = ctx.set_query(np.zeros(20, np.uint8), 1, -np.ones((5, 5)) + 3 * np.eye(5), {mode}, 3, 1, {ends}, 40, 0.5)
ctx.score_set(qid, sid)
windows = ctx.last_windows()
assert windows > 400
def upload(i, dtype):
    a = np.empty(fake.fake_upload(i, None), np.uint8)
    fake.fake_upload(i, a.ctypes.data_as(C.c_char_p))
    return a.view(dtype)
cs, start, slot, length = (upload(i, np.uint32) for i in range(4))
assert len(length) == windows and sorted(slot) == list(range(windows))
first = start[slot] == 0
if {split}:
    assert (np.diff(first.astype(int)) <= 0).all()
    assert (np.diff(length[first].astype(int)) <= 0).all() and (np.diff(length[~first].astype(int)) <= 0).all()
else:
    assert (np.diff(length.astype(int)) <= 0).all()
""")

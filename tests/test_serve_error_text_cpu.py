"""The context's error text belongs to its caller: a failure on the serving
thread reaches it through poll alone, on a runtime without a device."""
import pytest

from fake_device import fake_lib, run  # noqa: F401


@pytest.mark.parametrize("what", ["launch", "profile", "exact kernels"])
def test_text_of_the_caller_stays(fake_lib, what):  # noqa: F811
    run(fake_lib, f"""
import time
what = {what!r}
off = np.arange(301, dtype=np.uint64) * 40
sid = ctx.records_load(np.zeros(int(off[-1]), np.uint8), off)
gap = 1 if what[0] == "e" else 3  # linear gaps go to the exact kernels
qid = ctx.set_query(np.zeros(20, np.uint8), 1, -np.ones((5, 5)) + 3 * np.eye(5), native.ALGO_LOCAL, gap, 1, 15, 40,
                    0.5)
ctx.serve_start(sid)
fake.fake_refuse_func_attributes(what[0] == "l")
fake.fake_refuse_memory_to_other_threads(what[0] != "l")
try:
    ctx.free_query(qid + 100)
except native.IshGpuError:
    pass
text = ctx._L.ish_gpu_last_error(ctx._h)
ticket = ctx.submit(qid)
time.sleep(0.3)
assert ctx._L.ish_gpu_last_error(ctx._h) == text
try:
    assert ctx.poll(ticket, 10000) is None
except native.IshGpuError as e:
    assert "refused" in str(e) or what[0] == "p", e  # (a profile's failure has a text of its own)
else:
    assert False
fake.fake_refuse_memory_to_other_threads(0)
ctx.serve_stop()
""")

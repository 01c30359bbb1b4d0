"""A load or scoring call that finds memory short gets back what start finding
keeps between calls, on a runtime without a device."""
import pytest

from fake_device import fake_lib, run  # noqa: F401


@pytest.mark.parametrize("call", ["load", "score"])
def test_every_allocation_is_tried_again(fake_lib, call):  # noqa: F811
    run(fake_lib, f"""
def records(n):
    off = np.arange(n + 1, dtype=np.uint64) * 300
    return np.zeros(int(off[-1]), np.uint8), off
qid = ctx.set_query(np.zeros(20, np.uint8), 1, -np.ones((5, 5)) + 3 * np.eye(5), native.ALGO_LOCAL, 3, 1, 15, 40, 0.5)
kept = ctx.records_load(*records(50))
ctx.score_set(qid, kept)
for k in range(12):
    ctx.match_starts(qid, kept, np.arange(50), np.full(50, 299))  # leaves its buffers with the context
    if {call!r} == "load":
        ctx.set_option(native.OPT_FAULT_ALLOC, k)
        ctx.records_load(*records(100 * 2 ** (k % 6) + (0 if k < 6 else 4000)))  # larger than before: it allocates
    else:
        sid = ctx.records_load(*records(100 * 2 ** (k % 6) + (0 if k < 6 else 4000)))
        ctx.set_option(native.OPT_FAULT_ALLOC, k % 4)  # scores, ends, hits
        ctx.score_set(qid, sid)
    ctx.set_option(native.OPT_FAULT_ALLOC, -1)
""")

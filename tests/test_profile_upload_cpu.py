"""No kernel is launched while the profile, the parameters or the tables that it
reads may still be on their way to the device, on a runtime without a device."""
import pytest

from fake_device import fake_lib, run  # noqa: F401


@pytest.mark.parametrize("n", [100, 5000])
def test_first_launches_of_queries(fake_lib, n):  # noqa: F811
    out = run(fake_lib, f"""
from ish_gb300.scoring import ScoringMatrix
off = np.arange({n} + 1, dtype=np.uint64) * 90
buf = np.full(int(off[-1]), 1, np.uint8)
sid = ctx.records_load(buf, off)
m = ScoringMatrix(1)
def query(Q, algo, gap=3, ext=1, ends=12):
    return ctx.set_query(np.random.default_rng(Q).integers(0, 4, Q, dtype=np.uint8), 1, m.values, algo, gap, ext, ends, 2 * Q, 0.5)
def check(what):
    report = fake.fake_report().decode()
    assert report == "", (what, report)
for algo in (native.ALGO_SEMI_GLOBAL, native.ALGO_LOCAL):
    for kernel in (native.KERNEL_AUTO, native.KERNEL_PLAIN, native.KERNEL_EXACT):
        ctx.set_option(native.OPT_KERNEL, kernel)
        ctx.score(query(2, algo), buf, off)
        check("one-shot")
        ctx.score_set(query(40, algo), sid)
        check("set")
    ctx.set_option(native.OPT_KERNEL, native.KERNEL_AUTO)
    ctx.score_set(query(31, algo, 2, 2), sid)
    check("linear gaps")
    ctx.score_set(query(300, algo, 2, 2), sid)
    check("linear gaps, long")
    q = query(50, algo)
    ctx.score_set(q, sid)
    ctx.match_starts(q, sid, [0, 1], [50, 80])
    check("starts")
    ctx.score_multi([query(20, algo), query(90, algo), query(20, algo, 2, 2)], sid)
    check("batched")
    ctx.serve_start(sid)
    tickets = [ctx.submit(query(20, algo)), ctx.submit(query(20, algo, 2, 2))]
    while any(ctx.poll(t, 100) is None for t in tickets):
        pass
    ctx.serve_stop()
    check("serving")
ctx.records_load_raw(np.full(int(off[-1]), 65, np.uint8), off, 1)
check("encoding")
""")
    assert out.strip() == ""

"""A one-shot call that is refused for a code outside the alphabet writes none of
the caller's arrays, whichever it asks for, on a runtime without a device."""
import pytest

from fake_device import fake_lib, run  # noqa: F401


@pytest.mark.parametrize("n", [1, 4096, 4097])
def test_arrays_are_left_alone(fake_lib, n):  # noqa: F811
    run(fake_lib, f"""
off = np.arange({n} + 1, dtype=np.uint64) * 30
buf = np.zeros(int(off[-1]), np.uint8)
buf[17] = 5
qid = ctx.set_query(np.zeros(20, np.uint8), 1, -np.ones((5, 5)) + 3 * np.eye(5), native.ALGO_LOCAL, 3, 1, 15, 40, 0.5)
types = (C.c_int32, C.c_int32, C.c_int32, C.c_uint8, C.c_uint32, C.c_uint32)
for want in range(64):
    arrays = [np.full({n}, 7, np.dtype(t)) if want >> i & 1 else None for i, t in enumerate(types)]
    rc = ctx._L.ish_gpu_score(ctx._h, qid, native._p(buf, C.c_uint8), native._p(off, C.c_uint64), {n},
                              *(native._p(a, t) for a, t in zip(arrays, types)))
    assert rc == native.EINVAL, want
    assert b"code 5 >= the alphabet" in ctx._L.ish_gpu_last_error(ctx._h)
    assert all((a == 7).all() for a in arrays if a is not None), want
""")

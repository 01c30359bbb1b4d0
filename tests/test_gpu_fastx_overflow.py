"""Texts with more records than there is room for their bounds: the refused call
says how many there are, and the next one has them without a count on the host."""
import ctypes as C

import numpy as np
import pytest

from ish_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("records", [2, 3, 60_000])
def test_refused_call_counts_the_records(records, monkeypatch):
    sparse = b">long\n" + b"A" * 199_990 + b"\n"
    text = np.frombuffer(sparse * 40 + b"".join(b">%d\nACGTN\n" % i for i in range(records - 1)) + b">e\nA\n", np.uint8)
    total = 40 + records
    with native.Context(0) as c:
        for room in (0, 1, total - 1, total):
            sid, n = C.c_int32(), C.c_uint32()
            bnd = np.zeros((max(room, 1), 4), np.uint64)
            rc = c._L.ish_gpu_records_load_fastx(c._h, native._p(text, C.c_uint8), len(text), 1, C.byref(sid),
                                                 C.byref(n), native._p(bnd, C.c_uint64), room)
            assert (rc, n.value) == (native.OK if room == total else native.EOVERFLOW, total)
        room = 41 if records > 41 else total - 1
        monkeypatch.setattr(native, "_line_room", lambda buf: room)
        monkeypatch.delattr(np, "count_nonzero")
        _, n, bounds = c.records_load_fastx(text, 1)
        assert n == len(bounds) == total and bytes(text[int(bounds[-1, 0]):int(bounds[-1, 1])]) == b"e"

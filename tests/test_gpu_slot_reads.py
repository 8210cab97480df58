"""Reads of slots that are not neighbours: one wait for the stream (one per filling
of the pinned buffer where flows pass through it), the same flows as slot by slot."""
import ctypes

import numpy as np
import pytest

from pdflow import BatchSolver, scenes
from pdflow._lib import check, load

pytestmark = pytest.mark.gpu


def _waits(b):
    n = ctypes.c_ulonglong(0)
    check(load().pdflow_wait_count(b.handle, ctypes.byref(n)), "pdflow_wait_count")
    return n.value


@pytest.mark.parametrize("pin", [False, True])
@pytest.mark.parametrize("rows", [15, 60, 240])
def test_scattered_slots_wait_once(built_lib, rows, pin):
    """Flows of 15 and 60 rows pass through the handle's pinned buffer where the
    caller's memory is pageable, up to four of 60 rows at a time (256 KB); a longer
    run of those and everything else goes directly."""
    import torch
    n, N = 7, rows * rows * 4 // 3
    b = BatchSolver(rows, 320, 240, n)
    pairs = [scenes.make_pair(80 + k) for k in range(n)]
    for f in (0, 1):
        b.push_slots(range(n), np.stack([p[2 * f] for p in pairs]), np.stack([p[2 * f + 1] for p in pairs]))
    b.solve_slots(list(range(n)))

    def read(slots):
        out = [torch.full((len(slots), N), 7.0, pin_memory=pin) for _ in range(3)]
        sl = np.array(slots, np.uint32)
        before = _waits(b)
        check(load().pdflow_read_flow_slots(b.handle, len(slots), sl.ctypes.data_as(ctypes.c_void_p),
                                            *[ctypes.c_void_p(t.data_ptr()) for t in out]), "read")
        return torch.stack(out).numpy().view(np.uint32).copy(), _waits(b) - before

    one = [read([k])[0][:, 0] for k in range(n)]
    assert len({o.tobytes() for o in one}) == n
    for slots, fillings in (([5], 1), ([6, 2, 4], 1), ([0, 1, 5, 3], 1), ([1, 3, 5, 0, 6, 2, 4], 2),
                            ([4, 5, 6, 0, 1, 3], 2), (list(range(n)), 1), ([6, 0, 1, 2, 3, 4], 2)):
        got, waits = read(slots)
        assert waits == (fillings if rows == 60 and not pin else 1), (slots, waits)
        for j, k in enumerate(slots):
            assert np.array_equal(got[:, j], one[k]), (slots, k)
    b.close()

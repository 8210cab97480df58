"""Pinned host memory of a handle: none until a call has a use for it."""
import ctypes

import numpy as np
import pytest

from pdflow import BatchSolver, MixedBatch, Solver, scenes
from pdflow._lib import check, load

pytestmark = pytest.mark.gpu


def _pinned(s):
    n = ctypes.c_size_t(1)
    check(load().pdflow_pinned_bytes(s.handle, ctypes.byref(n)), "pdflow_pinned_bytes")
    return n.value


@pytest.mark.parametrize("rows,width,n", [(15, 320, 1), (240, 320, 1), (480, 640, 1), (60, 320, 4)])
def test_a_device_caller_pins_nothing(built_lib, rows, width, n):
    """Frames pushed from the device and flows copied on it: no pinned memory,
    neither at creation nor at the first pass."""
    import torch
    frames = [scenes.make_pair(20 + k, vga=width == 640) for k in range(n)]
    dev = [torch.from_numpy(np.stack([f[c] for f in frames])).cuda() for c in range(4)]
    out = [torch.empty(n, rows * rows * 4 // 3, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    b = BatchSolver(rows, width, width * 3 // 4, n)
    assert _pinned(b) == 0
    for f in (0, 2):
        b.push_raw_device(n, dev[f].data_ptr(), dev[f + 1].data_ptr())
    b.solve(n)
    check(load().pdflow_copy_flow_device(b.handle, n, *[o.data_ptr() for o in out]), "copy")
    torch.cuda.synchronize()
    assert _pinned(b) == 0
    want = np.stack(b.read_flow(n))   # now it has one
    assert _pinned(b) > 0
    assert np.array_equal(want.view(np.uint32), torch.stack(out).cpu().numpy().view(np.uint32))
    b.close()


def test_host_frames_and_flows_pin_at_first_use(built_lib):
    i1, z1, i2, z2 = scenes.make_pair(3)
    s = Solver(60, 320, 240).initializeCUDA()
    assert _pinned(s) == 0
    s.push_raw(i1, z1)
    frames = _pinned(s)
    assert frames >= 320 * 240 * 3
    s.push_raw(i2, z2)
    assert _pinned(s) == frames
    s.solveSceneFlowGPU()
    all_ = _pinned(s)
    assert all_ >= frames + 60 * 80 * 12
    s.solveSceneFlowGPU()
    assert _pinned(s) == all_
    s.freeGPUMemory()


def test_a_mixed_handle_pins_at_its_first_read(built_lib):
    rows = [60, 480]
    small, big = scenes.make_pair(4), scenes.make_pair(4, vga=True)
    m = MixedBatch(2)
    assert _pinned(m) == 0
    for f in (0, 1):
        m.push(rows, [small[2 * f], big[2 * f]], [small[2 * f + 1], big[2 * f + 1]])
    m.solve()
    assert _pinned(m) == 0
    for k in range(2):
        got = m.flow(k)
        s = Solver(rows[k], 640 if k else 320, 480 if k else 240).initializeCUDA()
        s.loadRGBDFrames(*(big if k else small))
        s.solveSceneFlowGPU()
        for a, w in zip(got, (s.dxp, s.dyp, s.dzp)):
            assert np.array_equal(a.view(np.uint32), w.view(np.uint32))
        s.freeGPUMemory()
    # its passing results are those of rows up to 120, not the whole arena's
    assert 60 * 80 * 12 <= _pinned(m) <= (256 << 10) + 4096
    m.close()


def test_handles_replaced_in_several_threads(built_lib):
    """Blocks of destroyed handles serve new ones: four threads that each replace
    handles of different sizes, the old one destroyed before or after the new one's
    first use, get every pair's own flow."""
    import threading
    kinds = [(60, 1), (15, 3), (60, 6), (30, 1)]
    pairs = [scenes.make_pair(30 + k) for k in range(6)]

    def solve(rows, n, shift, old=None):
        b = BatchSolver(rows, 320, 240, n)
        order = [pairs[(shift + k) % 6] for k in range(n)]
        for f in (0, 1):
            b.push_raw(np.stack([p[2 * f] for p in order]), np.stack([p[2 * f + 1] for p in order]))
        if old is not None:
            old.close()
        b.solve(n)
        return b, np.stack(b.read_flow(n)).view(np.uint32).copy()

    want = {}
    for rows, n in kinds:
        for shift in range(3):
            b, want[rows, n, shift] = solve(rows, n, shift)
            b.close()
    bad = []

    def work(t):
        old = None
        for rep in range(12):
            rows, n = kinds[(t + rep) % 4]
            if old is not None and rep % 2:
                old.close()
                old = None
            old, got = solve(rows, n, rep % 3, old)
            if not np.array_equal(got, want[rows, n, rep % 3]):
                bad.append((t, rep))
        old.close()

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    assert all(w.any() for w in want.values())

"""Frames and results that pass through a handle's pinned buffers (pageable memory
of the caller, up to a size) against the direct copies (pinned memory of the
caller): the same bits, whatever the caller does with its frames afterwards."""
import ctypes

import numpy as np
import pytest

from pdflow import BatchSolver, Solver, scenes
from pdflow._lib import check, load

pytestmark = pytest.mark.gpu


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("kind,rows", [("u16", 15), ("float", 60), ("rgb", 240)])
def test_frames_pageable_and_pinned(built_lib, kind, rows):
    import torch
    i1, z1, i2, z2 = scenes.make_pair(31)
    frames = [(i1, z1), (i2, z2)]
    if kind == "float":
        frames = [scenes.decode(*f) for f in frames]
    if kind == "rgb":
        frames = [(np.stack([i, i // 2, 255 - i], -1), z) for i, z in frames]
    call = {"u16": "pdflow_push_frame_u16", "float": "pdflow_push_frame", "rgb": "pdflow_push_frame_rgb8_mm"}[kind]
    extra = (0,) if kind == "rgb" else ()
    flows = []
    for pin in (False, True):
        s = Solver(rows, 320, 240).initializeCUDA()
        for rep in range(2):   # four frames: each buffer is used again
            for f in frames:
                ts = [torch.from_numpy(np.array(a)) for a in f]
                ts = [t.pin_memory() for t in ts] if pin else ts
                check(getattr(load(), call)(s.handle, *[_ptr(t) for t in ts], *extra), call)
                if pin:
                    s.synchronize()
                for t in ts:
                    t.zero_()
        s.solveSceneFlowGPU(read_back=False)
        out = [torch.full((rows * rows * 4 // 3,), 7.0, pin_memory=pin) for _ in range(3)]
        check(load().pdflow_read_flow(s.handle, *[_ptr(t) for t in out]), "pdflow_read_flow")
        flows.append(torch.stack(out).numpy().view(np.uint32).copy())
        s.freeGPUMemory()
    assert np.array_equal(flows[0], flows[1]) and flows[0].any()


@pytest.mark.parametrize("rows", [15, 60, 240])
def test_slots_read_in_runs(built_lib, rows):
    """Scattered, reversed and consecutive slots (up to four 60-row flows in a run
    pass, seven and the 240-row ones go directly) against every slot read by itself into pinned memory."""
    import torch
    n, N = 7, rows * rows * 4 // 3
    b = BatchSolver(rows, 320, 240, n)
    pairs = [scenes.make_pair(60 + k) for k in range(n)]
    for f in (0, 1):
        for k in (3, 0, 6, 1, 2, 5, 4):
            b.push_slots([k], pairs[k][2 * f][None], pairs[k][2 * f + 1][None])
    b.solve_slots(list(range(n)))
    one = []
    for k in range(n):
        out = [torch.zeros(N, pin_memory=True) for _ in range(3)]
        sl = np.array([k], np.uint32)
        check(load().pdflow_read_flow_slots(b._h, 1, sl.ctypes.data_as(ctypes.c_void_p), *[_ptr(t) for t in out]), "read")
        one.append(torch.stack(out).numpy().view(np.uint32).copy())
    for slots in ([0], [4, 5, 6, 0, 1, 3], [6, 5, 4], list(range(n))):
        got = np.stack(b.read_flow_slots(slots)).view(np.uint32)
        for j, k in enumerate(slots):
            assert np.array_equal(got[:, j], one[k]), (slots, k)
    assert len({o.tobytes() for o in one}) == n
    b.close()

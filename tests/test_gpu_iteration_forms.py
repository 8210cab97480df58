"""What the launch forms run, by launch counts and the planner's work."""
import ctypes

import numpy as np
import pytest

from pdflow import BatchSolver, MixedBatch, scenes
from pdflow._lib import check, load

pytestmark = pytest.mark.gpu


def _batch(rows, n, **kw):
    pairs = [scenes.make_pair(500 + k) for k in range(n)]
    b = BatchSolver(rows, 320, 240, n, **kw)
    for f in (0, 1):
        b.push_raw(np.stack([p[2 * f] for p in pairs]), np.stack([p[2 * f + 1] for p in pairs]))
    return b


def _launches(s):
    n = ctypes.c_uint(0)
    check(load().pdflow_last_solve_launches(s.handle, ctypes.byref(n)), "launches")
    return n.value


def _plans():
    n = ctypes.c_ulonglong(0)
    check(load().pdflow_strip_plan_count(ctypes.byref(n)), "plans")
    return n.value


@pytest.mark.parametrize("form", [5, 7, 8, 9])
def test_tiles_plan_no_strips(built_lib, form):
    """Only the strips' launches look for a plan of strips: 11 pairs of a size no
    other test uses, every level in a tile form chosen by hand."""
    b = _batch(240, 11, use_graph=False)
    for level in range(5):
        check(load().pdflow_set_level_form(b.handle, level, form, 0), "form")
    before = _plans()
    b.solve(11)
    b.synchronize()
    assert _plans() == before
    b.close()


def test_a_resident_level_is_probed_once(built_lib):
    """At 30x40 form 9 runs the level in one launch whatever the iterations per
    launch: its candidates are one, with one time."""
    b = _batch(30, 2)
    rep = b.autotune(2)
    times = rep[1]["ms_per_iter"][23:26]   # form 9 at 4, 6 and 8 iterations per launch
    assert times[0] is not None and times[0] == times[1] == times[2]
    b.close()
    m = MixedBatch(2)
    pairs = [scenes.make_pair(500 + k) for k in range(2)]
    for f in (0, 1):
        m.push([30, 30], [p[2 * f] for p in pairs], [p[2 * f + 1] for p in pairs])
    times = m.autotune(2)[1]["ms_per_iter"][23:26]
    assert times[0] is not None and times[0] == times[1] == times[2]
    m.close()


@pytest.mark.parametrize("form,iteration_launches", [(2, 25), (3, 25), (5, 25), (7, 25), (8, 25), (9, 25), (10, 1), (1, 1),
                                                     (0, 200)])
def test_a_batch_runs_15x20_in_the_form_asked_for(built_lib, form, iteration_launches):
    """100 iterations of three pairs at 15x20: tiles of four iterations a launch in
    every tile form, the default one launch; beside them gradients, two set-up
    launches and the median.  The same bits."""
    b = _batch(15, 3)
    b.solve(3)
    assert _launches(b) == 4 + 1
    want = np.stack(b.read_flow(3))
    check(load().pdflow_set_iteration_form(b.handle, form), "form")
    b.solve(3)
    assert _launches(b) == 4 + iteration_launches
    assert np.array_equal(np.stack(b.read_flow(3)).view(np.uint32), want.view(np.uint32))
    b.close()


@pytest.mark.parametrize("form,iteration_launches", [(5, 25), (8, 25), (9, 25), (10, 1)])
def test_a_mixed_batch_runs_15x20_in_the_form_asked_for(built_lib, form, iteration_launches):
    pairs = [scenes.make_pair(500 + k) for k in range(3)]
    m = MixedBatch(3)
    for f in (0, 1):
        m.push([15] * 3, [p[2 * f] for p in pairs], [p[2 * f + 1] for p in pairs])
    m.solve()
    want = [m.flow(k) for k in range(3)]
    check(load().pdflow_set_iteration_form(m.handle, form), "form")
    m.solve()
    assert _launches(m) == 4 + iteration_launches
    for k in range(3):
        for a, w in zip(m.flow(k), want[k]):
            assert np.array_equal(a.view(np.uint32), w.view(np.uint32))
    m.close()

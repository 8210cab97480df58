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

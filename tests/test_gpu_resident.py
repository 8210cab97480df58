"""The resident tiles (a level in one launch, a cluster per pair): bits against
the paired shared-memory tiles (form 5) at iteration counts around the
exchange period, batch sizes on both sides of the rule that picks them, and
through a slot map; and the 15x20 level's one launch for a batch."""
import numpy as np
import pytest

from pdflow import BatchSolver, default_params, scenes

pytestmark = pytest.mark.gpu


def _frames(n):
    pairs = [scenes.make_pair(70 + k, vga=False) for k in range(min(n, 4))]
    return [tuple(np.stack([pairs[k % len(pairs)][2 * f + c] for k in range(n)]) for c in (0, 1)) for f in (0, 1)]


def _solve(n, iters, forms, slots=None):
    p = default_params(60)
    for i, k in enumerate(iters):
        p.num_max_iter[i] = k
    s = BatchSolver(60, 320, 240, n, p)
    for level, form in enumerate(forms):
        s.set_level_form(level, form)
    for intensity, depth in _frames(n if slots is None else len(slots)):
        if slots is None:
            s.push_raw(intensity, depth)
        else:
            s.push_slots(slots, intensity, depth)
    if slots is None:
        s.solve(n)
        out = np.stack(s.read_flow(n))
    else:
        s.solve_slots(slots)
        out = np.stack(s.read_flow_slots(slots))
    s.close()
    return out.view(np.uint32)


@pytest.mark.parametrize("iters", [(1, 1, 1), (2, 3, 4), (3, 5, 8), (4, 13, 97)])
@pytest.mark.parametrize("n", [1, 3, 21])
def test_resident_levels_equal_the_paired_tiles(built_lib, n, iters):
    ref = _solve(n, iters, (5, 5, 5))
    assert np.array_equal(_solve(n, iters, (-1, -1, -1)), ref)   # the default forms
    assert np.array_equal(_solve(n, iters, (1, 9, 9)), ref)      # one launch, resident or deep tiles


def test_resident_levels_through_a_slot_map(built_lib):
    slots = [4, 0, 2]
    assert np.array_equal(_solve(6, (9, 9, 9), (-1, -1, -1), slots), _solve(6, (9, 9, 9), (5, 5, 5), slots))

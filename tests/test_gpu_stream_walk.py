"""The streamed tiles' and strips' region walk where a launch has fewer regions
than CTAs, exactly one a CTA, or a few: the producer's first, last and only
region.  Bits against the paired shared-memory tiles (form 5)."""
import numpy as np
import pytest

from pdflow import BatchSolver, scenes

pytestmark = pytest.mark.gpu

ROWS = 120


def _solve(n, form, kk, frames):
    s = BatchSolver(ROWS, 320, 240, n)
    for level in range(1, 4):
        s.set_level_form(level, form, kk)
    for intensity, depth in frames:
        s.push_raw(intensity, depth)
    s.solve(n)
    out = np.stack(s.read_flow(n))
    s.close()
    return out.view(np.uint32)


@pytest.mark.parametrize("n", [1, 3, 31])
def test_walks_equal_the_paired_tiles(built_lib, n):
    pairs = [scenes.make_pair(40 + k, vga=False) for k in range(min(n, 3))]
    frames = [tuple(np.stack([pairs[k % len(pairs)][2 * f + c] for k in range(n)]) for c in (0, 1)) for f in (0, 1)]
    ref = _solve(n, 5, 4, frames)
    for form, kk in ((8, 4), (8, 1), (9, 8), (9, 5), (10, 4), (10, 3), (10, 1)):
        assert np.array_equal(_solve(n, form, kk, frames), ref), (form, kk)


@pytest.mark.parametrize("n", [5, 10])
def test_planned_strip_units_equal_the_paired_tiles(built_lib, n):
    """Batch sizes whose 240x320 level runs strips cut by when the queue ends
    (5: every strip in 3 pieces; 10: two runs of different pieces)."""
    pairs = [scenes.make_pair(60 + k, vga=False) for k in range(3)]
    frames = [tuple(np.stack([pairs[k % 3][2 * f + c] for k in range(n)]) for c in (0, 1)) for f in (0, 1)]

    def solve(forms):
        s = BatchSolver(240, 320, 240, n)
        for level, form in forms.items():
            s.set_level_form(level, form)
        for intensity, depth in frames:
            s.push_raw(intensity, depth)
        s.solve(n)
        out = np.stack(s.read_flow(n))
        s.close()
        return out.view(np.uint32)

    assert np.array_equal(solve({}), solve({level: 5 for level in range(5)}))

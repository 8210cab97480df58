"""Mixed batches whose small steps run as one launch with each pair's own
iteration count, against the same batch with every step as tiles (iteration form
8): same bits, on both sides of the rule's line (20 pairs at 60x80)."""
import numpy as np
import pytest

from pdflow import MixedBatch, scenes
from pdflow._lib import check, load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [[15], [30, 15, 60, 120, 60, 30], [60] * 19 + [120], [60, 120, 30] * 8 + [15]])
def test_whole_steps_equal_tiles(built_lib, rows):
    pairs = [scenes.make_pair(300 + k, n_objects=1 + k % 5) for k in range(len(rows))]
    flows = []
    for form in (10, 8):
        b = MixedBatch(len(rows) + 1)
        check(load().pdflow_set_iteration_form(b.handle, form), "pdflow_set_iteration_form")
        for f in (0, 1):
            b.push(rows, [p[2 * f] for p in pairs], [p[2 * f + 1] for p in pairs])
        for _ in range(2):
            b.solve()
        flows.append([np.stack(b.flow(k)).view(np.uint32).copy() for k in range(len(rows))])
        b.close()
    for k, (x, y) in enumerate(zip(*flows)):
        assert x.any() and np.array_equal(x, y), (k, rows[k])

"""Launches that start while the kernel before them ends: solves and pushes
queued without a wait between them, through graphs and as plain launches, give
the bits of solves that are waited for one by one."""
import numpy as np
import pytest

from pdflow import BatchSolver, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("rows,n", [(15, 1), (60, 3), (240, 1), (240, 8)])
def test_queued_solves_equal_waited_ones(built_lib, rows, n, graph):
    import torch
    frames = [[torch.from_numpy(np.stack([scenes.make_pair(40 + k + 7 * f)[j] for k in range(n)])).cuda()
               for j in (0, 1)] for f in range(3)]
    b = BatchSolver(rows, 320, 240, n, use_graph=graph)
    N = rows * rows * 4 // 3

    def push(f):
        b.push_raw_device(n, frames[f][0].data_ptr(), frames[f][1].data_ptr())

    torch.cuda.synchronize()
    want = {}
    push(0)
    for f in (1, 2, 0, 1):
        push(f)
        b.solve(n)
        want[f] = np.stack(b.read_flow(n)).view(np.uint32).copy()
    assert want[0].any() and not np.array_equal(want[0], want[1])
    for last in (2, 0, 1):
        for rep in range(4):   # twelve pushes and solves behind one another, then one read
            for f in ((last + 1) % 3, (last + 2) % 3, last):
                push(f)
                b.solve(n)
        got = np.stack(b.read_flow(n)).view(np.uint32)
        assert got.shape == (3, n, N)
        assert np.array_equal(got, want[last]), last
    b.close()

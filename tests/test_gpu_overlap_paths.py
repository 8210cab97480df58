"""Launches that start while the kernel before them ends, on the paths beside the
plain batch: slot solves, mixed batches and the learned warm start, queued without a
wait between them, give the bits of solves that are waited for one by one."""
import numpy as np
import pytest

from pdflow import BatchSolver, MixedBatch, Net, load_weights, scenes

pytestmark = pytest.mark.gpu


def _stack(pairs, f):
    return np.stack([p[2 * f] for p in pairs]), np.stack([p[2 * f + 1] for p in pairs])


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("rows,slots", [(60, [2, 0]), (240, [3, 1, 4])])
def test_queued_slot_solves(built_lib, rows, slots, graph):
    frames = [[scenes.make_pair(40 + k + 7 * f)[:2] for k in range(len(slots))] for f in range(3)]

    def push(b, f):
        b.push_slots(slots, np.stack([x[0] for x in frames[f]]), np.stack([x[1] for x in frames[f]]))

    def solve(order, wait):
        b = BatchSolver(rows, 320, 240, 5, use_graph=graph)
        push(b, order[0])
        for f in order[1:]:
            push(b, f)
            b.solve_slots(slots)
            if wait:
                b.synchronize()
        got = np.stack(b.read_flow_slots(slots)).view(np.uint32).copy()
        b.close()
        return got

    for order in ([0, 1, 2, 0, 1], [2, 1, 0, 2]):
        want = solve(order, True)
        assert want.any()
        for _ in range(3):
            assert np.array_equal(solve(order, False), want)


@pytest.mark.parametrize("graph", [True, False])
def test_queued_mixed_solves(built_lib, graph):
    rows = [60, 15, 240, 120, 30]
    frames = [[scenes.make_pair(40 + k + 7 * f)[:2] for k in range(len(rows))] for f in range(3)]

    def solve(wait):
        m = MixedBatch(len(rows), use_graph=graph)
        for q, f in enumerate((0, 1, 2, 0)):
            m.push(rows, [x[0] for x in frames[f]], [x[1] for x in frames[f]])
            if q:
                for _ in range(3):   # the same frames again, behind the solve before
                    m.solve()
                    if wait:
                        m.synchronize()
        got = [np.stack(m.flow(k)).view(np.uint32).copy() for k in range(len(rows))]
        m.close()
        return got

    want = solve(True)
    for _ in range(3):
        for a, w in zip(solve(False), want):
            assert w.any() and np.array_equal(a, w)


@pytest.mark.parametrize("n", [2, 17])
def test_queued_learned_solves(built_lib, n):
    """2 pairs run the network's im2col kernels, 17 its gathers."""
    frames = [_stack([scenes.make_pair(40 + k + f) for k in range(n)], 0) for f in range(3)]
    net = Net(n)
    net.set_params(load_weights())

    def solve(wait):
        b = BatchSolver(120, 320, 240, n)
        for q, f in enumerate((0, 1, 2, 0)):
            b.push_raw(*frames[f])
            if q:
                for _ in range(2):
                    b.solve_learned(n, net, 0.75, 0.01)
                    if wait:
                        b.synchronize()
        got = np.stack(b.read_flow(n)).view(np.uint32).copy()
        b.close()
        return got

    want = solve(True)
    assert want.any()
    for _ in range(3):
        assert np.array_equal(solve(False), want)
    net.close()

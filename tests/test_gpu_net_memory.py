"""Device memory of the warm-start network's workspaces."""
import pytest

from pdflow import Net, _lib

pytestmark = pytest.mark.gpu


def _bytes(n):
    net = Net(n)
    size = _lib.load().pdflow_net_device_bytes(net.handle)
    net.close()
    return size


def test_im2col_matrix_only_for_the_batches_that_use_it(built_lib):
    """Forward passes of fewer than 16 inputs read an im2col matrix of the widest
    layer (4800 pixels x 9 * 48 bf16 values an input); larger ones gather.  So an
    input more costs that much less beyond 15 inputs than below, to a thousandth
    (the loss's block sums round)."""
    small, large = (_bytes(12) - _bytes(4)) / 8, (_bytes(64) - _bytes(32)) / 32
    matrix = 4800 * 9 * 48 * 2
    assert abs(small - large - matrix) <= matrix / 1000
    assert _bytes(15) + 49 * (large + 64) >= _bytes(64)

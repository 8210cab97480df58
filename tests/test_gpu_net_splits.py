"""The weight and bias gradients of the warm-start network where their sum over the
pixels is split over the most CTAs."""
import numpy as np
import pytest

from oracle import net_oracle as no
from pdflow import Net

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 64])
def test_gradients_of_copies_are_one_input_s(built_lib, n):
    """n copies of one input, n a power of two: the loss's 1 / count scales every
    output gradient, and so every bf16 gradient of the backward pass, by exactly 1 / n,
    and each parameter's gradient sums the n copies of one input's terms: the same sum
    in another order and split (one input's is compared with the oracle elsewhere).
    An FP32 sum rounds each partial sum once: at most 300 steps serial in a split, 76
    partials added in order and 8 of those: 400 * 2^-23 = 4.8e-5 of the
    largest partial sum, which stays near the sum itself where terms cancel like
    noise; 5e-4 of the layer's norm is taken.  A split left out or taken twice
    moves it by 1 / 600 and more."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    inp = np.zeros((1, 4, no.HW), np.float32)
    inp[:, 0:2] = rng.uniform(0, 255, size=(1, 2, no.HW))
    inp[:, 2:4] = rng.uniform(0.8, 4.0, size=(1, 2, no.HW))
    inp[:, 2][rng.random((1, no.HW)) < 0.05] = 0
    label = (rng.normal(size=(1, 3, no.HW)) * np.array([1, 1, 0.02])[None, :, None]).astype(np.float32)
    params = no.init_params(33)
    grads = []
    for m in (1, n):
        net = Net(m)
        net.set_params(params)
        x = torch.from_numpy(np.repeat(inp, m, 0)).cuda()
        y = torch.from_numpy(np.repeat(label, m, 0)).cuda()
        grads.append(net.gradients(m, x.data_ptr(), y.data_ptr())[1].astype(np.float64))
        net.close()
    one, many = grads
    for i, c in enumerate(no.GRAPH.convs):
        for lo, count in ((c["woff"], c["cout"] * c["K"]), (c["boff"], c["cout"])):
            a, b = one[lo:lo + count], many[lo:lo + count]
            assert np.linalg.norm(a) > 0
            assert np.linalg.norm(b - a) <= 5e-4 * np.linalg.norm(a), (i, lo)

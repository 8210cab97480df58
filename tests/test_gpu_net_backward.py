"""The warm-start network's backward kernels at the batch sizes where their
launches change shape."""
import numpy as np
import pytest

from oracle import net_oracle as no
from pdflow import Net

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch(built_lib):
    return pytest.importorskip("torch")


def _batch(seed, n):
    rng = np.random.default_rng(seed)
    inp = np.zeros((n, 4, no.HW), np.float32)
    inp[:, 0:2] = rng.uniform(0, 255, size=(n, 2, no.HW))
    inp[:, 2:4] = rng.uniform(0.8, 4.0, size=(n, 2, no.HW))
    inp[:, 2][rng.random((n, no.HW)) < 0.05] = 0
    label = (rng.normal(size=(n, 3, no.HW)) * np.array([1, 1, 0.02])[None, :, None]).astype(np.float32)
    return inp, label


@pytest.mark.parametrize("n", [1, 2, 17, 64])
def test_head_bias_gradient_is_the_sum_of_the_output_gradients(torch, n):
    """db of the head = the sum over valid pixels of bf16(2 (out - label) / (3
    count)), from the network's own forward output.  An FP32 sum of N terms in
    a tree of depth d is off by at most d * 2^-24 of the sum of magnitudes;
    here at most 64 serial terms a thread, then 6 + 38 + 4 levels: 112 * 2^-24 =
    6.7e-6.  A term's input differs by the FP32 rounding of out * 20 and of the
    product (a few 2^-24), which flips its bf16 rounding (2^-8) in about one
    term in 2^14: 3e-7 on average, far below the bound taken, 2e-5."""
    net = Net(n, seed=3)
    net.set_params(no.init_params(12))
    inp, label = _batch(n, n)
    d_in, d_lab = torch.from_numpy(inp).cuda(), torch.from_numpy(label).cuda()
    out = torch.zeros((n, 3, no.HW), dtype=torch.float32, device="cuda")
    net.forward(n, d_in.data_ptr(), out.data_ptr())
    _, g = net.gradients(n, d_in.data_ptr(), d_lab.data_ptr())
    net.close()
    head = no.GRAPH.convs[-1]
    scale = np.array([1.0, 1.0, 20.0])[None, :, None]
    d = (out.cpu().numpy().astype(np.float64) - label) * scale * (inp[:, 2:3] > 0)
    terms = no.bf16((2 * d / (3 * int((inp[:, 2] > 0).sum()))).astype(np.float32)).astype(np.float64)
    got = g[head["boff"]:head["boff"] + 3].astype(np.float64)
    assert np.all(np.abs(got - terms.sum((0, 2))) <= 2e-5 * np.abs(terms).sum((0, 2)))


@pytest.mark.parametrize("n", [1, 5])
def test_gradients_against_the_oracle_at_ragged_pixel_counts(torch, n):
    """1 and 5 inputs: the deep levels' pixel counts (80 and 400 at 10x8) are no
    multiples of the GEMMs' 128 rows or of their split of the pixels.  Same
    bound as for two inputs: well inside what bf16 rounding itself moves."""
    net = Net(n, seed=3)
    p = no.init_params(21)
    net.set_params(p)
    inp, label = _batch(30 + n, n)
    d_in, d_lab = torch.from_numpy(inp).cuda(), torch.from_numpy(label).cuda()
    loss, g = net.gradients(n, d_in.data_ptr(), d_lab.data_ptr())
    net.close()
    rloss, rq = no.NetOracle(p, quantize=True).loss_and_grads(inp, label)
    _, rf = no.NetOracle(p, quantize=False).loss_and_grads(inp, label)
    assert abs(loss - rloss) <= 1e-5 * rloss
    rel = lambda x, y: np.linalg.norm(x - y) / max(np.linalg.norm(y), 1e-30)
    for i, c in enumerate(no.GRAPH.convs):
        lo, hi = c["woff"], c["woff"] + c["cout"] * c["K"]
        e_gpu, e_bf16 = rel(g[lo:hi].astype(np.float64), rq[lo:hi]), rel(rq[lo:hi], rf[lo:hi])
        assert e_gpu <= 0.75 * e_bf16 + 2e-3, (i, e_gpu, e_bf16)

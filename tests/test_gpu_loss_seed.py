"""The gradient of the loss at the network's output, rounded to f32 and to bf16, is
that of the f64 expression, value for value.

With all parameters zero the output is zero, e = -target, and the gradient of the
last layer's first bias is the sum over the pixels of the bf16 values, which the
inputs here make exact in f32, as they make the sums behind the mean and the
Laplacian exact in f64 in any order; so NumPy's f64 gives the expected sum to the
bit.  The weights put one pixel's value a few 2^-52 from the edge between two f32
values that bf16 rounds apart, where the last bits of the f64 value decide."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _bf16(x):
    return torch.from_numpy(np.asarray(x, np.float32)).to(torch.bfloat16).double().numpy()


def _seed_sum(e, w_p, w_r):
    """sum of bf16(f32(dL/dout)) of one image, in f64"""
    e = e.astype(np.float64)

    def lap(f):
        return np.roll(f, 1, 1) + np.roll(f, -1, 1) + np.roll(f, 1, 0) + np.roll(f, -1, 0) - 4.0 * f

    v = w_p * (e - e.sum() / e.size)
    if w_r:
        v = v + w_r * lap(lap(e).astype(np.float32).astype(np.float64))
    return _bf16((2.0 / e.size * v).astype(np.float32)).sum()


@pytest.fixture(scope="module")
def net(fs):
    g = fs.PressureGuess(seed=1)
    g.set_params(np.zeros_like(g.get_params()))
    yield g
    g.close()


def _device(net, e, w_p, w_r):
    net.set_loss(w_p, w_r)
    z = np.zeros((1, *e.shape), np.float32)
    _, grad = net.loss_grad(z, z, -e[None])
    return float(grad[-16])


@pytest.mark.parametrize("k", range(1, 17))
@pytest.mark.parametrize("side", [-3, -1, 1, 3])
def test_next_to_a_rounding_edge(net, k, side):
    # X w = the middle of the f32 values t and t + 2^-23, side 2^-52 beside it; t is
    # halfway between two bf16 values, the lower one even
    X = np.float32(1.0 + (8 * k + 3) / 1024.0 + 2.0 ** -20 * k)
    t = 1.0 + (4 * k + 1) / 256.0
    w = (t + 2.0 ** -24) / float(X)
    want = t + 2.0 ** -24 + side * 2.0 ** -52
    for _ in range(8):  # the f64 product on the wanted side of the middle
        if (float(X) * w - want) * side >= 0:
            break
        w = np.nextafter(w, np.inf if side > 0 else 0.0)
    assert (float(X) * w - (t + 2.0 ** -24)) * side > 0
    e = np.zeros((8, 8), np.float32)
    e[2, 3], e[5, 1], e[6, 6] = X, -1.0, -(X - np.float32(1.0))
    assert e.astype(np.float64).sum() == 0.0
    assert _device(net, e, 32.0 * w, 0.0) == _seed_sum(e, 32.0 * w, 0.0)


@pytest.mark.parametrize("shape", [(8, 8), (16, 40), (32, 32)])
@pytest.mark.parametrize("weights", [(1.3, 0.0), (0.05, 1.0), (0.0, 0.7), (3e-27, 1e-27), (1e-32, 3e-33), (1e9, 1e8)])
def test_values_of_all_sizes(net, shape, weights):
    rng = np.random.default_rng(shape[1])
    # multiples of 2^-18 below 1 in size: exact sums; many cells that cancel
    e = (rng.integers(-2 ** 18, 2 ** 18, shape) * rng.choice([0.0, 2.0 ** -6, 1.0], shape)).round() / 2.0 ** 18
    e = e.astype(np.float32)
    got, ref = _device(net, e, *weights), _seed_sum(e, *weights)
    # the device adds the bf16 values in f32: N 2^-24 of their sum of sizes
    scale = 2.0 * (2 * weights[0] + 64 * weights[1])
    assert abs(got - ref) <= e.size * 2.0 ** -24 * scale, (got, ref)

"""The loss of a training step against NumPy in float64, at image shapes that
cut the strips of its passes (30 columns, 8 or 32 rows a warp) and on values
that are widened to float64 in two ways (normal numbers; zeros and subnormals).

Both sides sum the same float64 terms, all of one sign, in other orders: at most
N 2^-53 = 1.1e-11 of the sum for the 1e5 cells here; 2e-11."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 8, 8), (3, 8, 24), (2, 16, 32), (1, 40, 64), (1, 72, 1032), (40, 32, 64)])
@pytest.mark.parametrize("weights", [(1.0, 0.0), (0.1, 1.0), (0.0, 2.0)])
def test_loss_value(fs, shape, weights):
    B, H, W = shape
    rng = np.random.default_rng(H * 10000 + W)
    div, tgt = rng.standard_normal((2, B, H, W)).astype(np.float32)
    tgt[rng.random(tgt.shape) < 0.1] = 0.0
    tgt[rng.random(tgt.shape) < 0.1] = 1e-41
    tgt[rng.random(tgt.shape) < 0.1] *= 1e-36
    mask = np.zeros_like(div)
    g = fs.PressureGuess(seed=31)
    g.set_loss(*weights)
    loss, grad = g.loss_grad(div, mask, tgt)
    e = g.predict(div, mask).cpu().numpy().astype(np.float64) - tgt.astype(np.float64)
    lap = np.roll(e, 1, 1) + np.roll(e, -1, 1) + np.roll(e, 1, 2) + np.roll(e, -1, 2) - 4.0 * e
    ec = e - e.mean(axis=(1, 2), keepdims=True)
    ref = weights[0] * np.mean(ec * ec) + weights[1] * np.mean(lap * lap)
    assert abs(loss - ref) <= 2e-11 * ref, (loss, ref)
    assert torch.isfinite(grad).all()
    g.close()


@pytest.mark.parametrize("size", [1e25, 1e29, 1e31])
def test_large_targets(fs, size):
    """Either side of the size (1e30) above which the gradient is formed in
    float64: against targets of 1 the gradient of this loss, which then hardly
    depends on the network's output, scales with the targets."""
    B, H, W = 1, 24, 40
    rng = np.random.default_rng(5)
    div, tgt = rng.standard_normal((2, B, H, W)).astype(np.float32)
    tgt *= np.float32(1e6)
    mask = np.zeros_like(div)
    g = fs.PressureGuess(seed=31)
    g.set_loss(0.1, 1.0)
    f = np.float32(2.0) ** int(np.log2(size / 1e6))  # a power of two: the same significands
    loss, grad = g.loss_grad(div, mask, tgt)
    grad = grad.cpu().numpy().astype(np.float64)
    loss_f, grad_f = g.loss_grad(div, mask, tgt * f)
    grad_f = grad_f.cpu().numpy().astype(np.float64) / float(f)
    # the output is 1e-6 of the targets: so is the difference of the errors; the
    # bf16 rounding of a few seeds goes the other way (1e-6 of them by 2^-9)
    assert abs(loss_f / float(f) ** 2 - loss) <= 1e-5 * loss
    assert np.linalg.norm(grad_f - grad) <= 1e-3 * np.linalg.norm(grad)
    g.close()

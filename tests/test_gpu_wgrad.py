"""The tensor-core weight gradients (fs_wgrad.cuh) at image shapes that cut
their tiles: rows and pixels left over, images narrower than a tile, single
rows and pixels on the coarse levels, several images.

The network is periodic, so an image repeated along x or y has the same
activations in every copy, an activation gradient of exactly 1/copies (the loss
is a mean; copies is a power of two) and the same parameter gradient -- summed
over other tiles, in another order.  f32 sums of up to ~1e3 terms per
accumulator differ by ~6e-8 sqrt(1e3) = 2e-6 of the sum; 2e-5 per layer.
Against the float64 restatement: test_gpu_guess.py."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import guess_oracle as G  # noqa: E402


@pytest.mark.parametrize("shape", [(1, 8, 8), (3, 8, 24), (1, 24, 136), (2, 40, 264), (1, 136, 48), (1, 8, 1032)])
def test_gradient_of_repeated_image(fs, shape):
    B, H, W = shape
    rng = np.random.default_rng(H * 10000 + W)
    div, tgt = rng.standard_normal((2, B, H, W)).astype(np.float32)
    mask = (rng.random((B, H, W)) > 0.8).astype(np.float32)
    g = fs.PressureGuess(seed=21)
    g.set_loss(0.1, 1.0)

    def grad(ry, rx):
        return g.loss_grad(*(np.tile(a, (1, ry, rx)) for a in (div, mask, tgt)))[1]

    one = grad(1, 1)
    assert torch.equal(one, grad(1, 1))  # partial sums are added in a fixed order
    one = one.cpu().numpy().astype(np.float64)
    for ry, rx in ((1, 2), (2, 1), (4, 4)):
        many = grad(ry, rx).cpu().numpy().astype(np.float64)
        k = 0
        for name, ci, co, _ in G.LAYERS:
            n = ci * co * 9 + co
            a, b = one[k:k + n], many[k:k + n]
            assert np.linalg.norm(a) > 0 and np.linalg.norm(a - b) <= 2e-5 * np.linalg.norm(a), (name, ry, rx)
            k += n
    g.close()

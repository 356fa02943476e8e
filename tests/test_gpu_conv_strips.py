"""The convolutions' walk over strips of rows and their fused epilogues
(fs_conv.cu) through the whole network, where strips and tiles are cut: rows
and pixels left over, images narrower than a tile or of one coarse pixel,
several images, several strips per CTA and several tiles per strip.

A pixel's sum is accumulated in one order wherever the pixel lies, and the
network is periodic, so an image repeated along x, y or the batch gives the
same output in every copy, to the bit.  One copy is checked against the float64
restatement, which rounds to bf16 where the device does (the tolerance of
test_gpu_guess.py: the occasional rounding that goes the other way)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import guess_oracle as G  # noqa: E402


def rnd(x):
    return torch.from_numpy(np.asarray(x, np.float32)).to(torch.bfloat16).double().numpy()


# repeats: (batch, y, x)
@pytest.mark.parametrize("shape, repeats", [
    ((1, 8, 8), [(400, 1, 1), (1, 16, 17)]),
    ((2, 8, 136), [(200, 1, 1), (3, 5, 1)]),
    ((1, 24, 120), [(1, 1, 9), (1, 40, 1)]),
    ((1, 40, 264), [(1, 3, 4), (101, 1, 1)]),
    ((1, 1032, 8), [(1, 1, 31), (3, 1, 1)]),
])
def test_output_of_repeated_image(fs, shape, repeats):
    B, H, W = shape
    rng = np.random.default_rng(H * 10000 + W)
    div = rng.standard_normal((B, H, W)).astype(np.float32)
    mask = (rng.random((B, H, W)) > 0.8).astype(np.float32)
    g = fs.PressureGuess(seed=23)
    one = g.predict(div, mask).cpu().numpy()
    ref, _ = G.forward(g.get_params().astype(np.float64), G.make_input(div.astype(np.float64), mask.astype(np.float64)),
                       rnd)
    assert np.linalg.norm(one - ref) <= 2e-2 * np.linalg.norm(ref)
    for r in repeats:
        many = g.predict(np.tile(div, r), np.tile(mask, r)).cpu().numpy()
        np.testing.assert_array_equal(many, np.tile(one, r))
    g.close()

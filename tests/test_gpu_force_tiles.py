"""The tiled forcing kernels (k_forcing, k_band_apply) against the oracle at
grids that cut their tiles and with counts that cut their batches of modes (8)
and of ky values (32).

Tolerance: an argument of up to ~60 rad rounds to 4e-6, as does its cosine; the
errors of the modes are independent, so the sums' relative L2 error is that or
less: 1e-5 (band: the tables are made in float64, 1e-6)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / np.linalg.norm(b))


@pytest.mark.parametrize("n", [8, 33, 64, 100, 136])
@pytest.mark.parametrize("count", [1, 7, 8, 9, 24])
def test_modes(fs, O, n, count):
    rng = np.random.default_rng(n * 100 + count)
    modes = [(float(kx), float(ky), float(ph)) for kx, ky, ph in
             zip(rng.integers(-9, 10, count), rng.integers(1, 10, count), rng.uniform(0, 6, count))]
    s = fs.GPUFluidSolver(n=n)
    s.upload_velocity(np.zeros(n * n), np.zeros(n * n))
    s.set_forcing(modes, amplitude=2.0, phase_drift=0.3)
    s.run_stage("forcing", 0.01)
    u, v = s.read_velocity()
    s.destroy()
    eu, ev = np.zeros((2, n * n))
    arr = (O.Mode * count)(*[O.Mode(*m) for m in modes])
    O.lib().fso_forcing_modes(O.grid(n), O._p(eu), O._p(ev), arr, count, 2.0, 0.0, 0.0, 0.01)
    assert np.linalg.norm(np.hypot(np.ravel(u) - eu, np.ravel(v) - ev)) <= 1e-5 * np.linalg.norm(np.hypot(eu, ev))


@pytest.mark.parametrize("n", [32, 66, 100, 130])
@pytest.mark.parametrize("kind, kf, width", [("gaussian", 3.0, 1.0), ("gaussian", 14.0, 0.8), ("gaussian", 33.0, 0.4),
                                             ("reference", 28.0, 2.0)])
def test_band(fs, O, n, kind, kf, width):
    s = fs.GPUFluidSolver(n=n)
    s.upload_velocity(np.zeros(n * n), np.zeros(n * n))
    s.set_band_forcing(kind, kf=kf, width=width, amplitude=0.4, seed=11)
    s.run_stage("forcing", 0.01)
    u, v = s.read_velocity()
    s.destroy()
    eu, ev = np.zeros((2, n * n))
    if kind == "reference":
        O.band_forcing(O.grid(n), eu, ev, kf, width, 0.4, 11, 0.01)
    else:
        O.gauss_band_forcing(O.grid(n), eu, ev, kf, width, 0.4, 11, 0, 0.01)
    assert rel(u, eu) <= 1e-6 and rel(v, ev) <= 1e-6

"""The flat solvers' fused sweeps (fs_flat.cu) against one pass per sweep or
colour (kernel_variant 1): the same arithmetic per cell, so equal bit for bit
at every grid shape, sweep count and start."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one cell to several periods in a region, tile edges and remainders of both
# regions (tiles of 40 and 104 columns; 200000 cells is where the larger takes over)
SHAPES = [(2, 2), (3, 5), (6, 2), (40, 40), (41, 39), (64, 64), (130, 70), (333, 500), (334, 500), (446, 448),
          (450, 446), (447, 449), (1042, 198), (2080, 121)]


def pressures(fs, nx, ny, **kw):
    rng = np.random.default_rng(nx * 10007 + ny)
    u, v = rng.standard_normal((2, nx * ny))
    out = []
    for variant in (0, 1):
        s = fs.GPUFluidSolver(nx=nx, ny=ny, lx=2.0, ly=2.0 * ny / nx, kernel_variant=variant, **kw)
        s.upload_velocity(u, v)
        s.run_stage("divergence", 0.01)
        got = []
        for _ in range(2):  # the second starts from the first's result with warm_start
            s.run_stage("pressure", 0.01)
            got.append(s.read_field("pressure"))
        s.step(1e-3)
        out.append(got + list(s.read_velocity()))
        s.destroy()
    return out


@pytest.mark.parametrize("solver", ["jacobi", "red-black"])
@pytest.mark.parametrize("nx,ny", SHAPES)
def test_fused_sweeps_equal_one_pass_per_sweep(fs, nx, ny, solver):
    for iterations, kw in ((1, {}), (12, {"relax": 0.8}), (25, {"warm_start": True}), (7, {"precision": "mixed"}),
                           (0, {})):
        a, b = pressures(fs, nx, ny, pressure_solver=solver, pressure_iterations=iterations, **kw)
        for x, y in zip(a, b):
            assert np.array_equal(x, y), (iterations, kw)


@pytest.mark.parametrize("solver", ["jacobi", "red-black"])
def test_non_finite_right_hand_side_spreads_alike(fs, solver):
    n = 96
    u, v = np.zeros((2, n * n))
    u[5 * n + 7], v[60 * n + 90] = np.inf, np.nan
    out = []
    for variant in (0, 1):
        s = fs.GPUFluidSolver(n=n, pressure_solver=solver, pressure_iterations=15, kernel_variant=variant)
        s.upload_velocity(u, v)
        s.run_stage("divergence", 0.01)
        s.run_stage("pressure", 0.01)
        out.append(s.read_field("pressure"))
        s.destroy()
    assert np.array_equal(out[0], out[1], equal_nan=True)


@pytest.mark.parametrize("solver", ["jacobi", "red-black"])
@pytest.mark.parametrize("nx,ny", [(24, 24), (23, 48), (256, 256), (264, 265), (384, 384), (416, 352)])
def test_launch_depths_equal_one_pass_per_sweep(fs, nx, ny, solver):
    """20, 16 and 12 sweeps a launch, by the CTAs that they make of the grid."""
    out = []
    for variant in (0, 1):
        rng = np.random.default_rng(nx * 1000 + ny)
        u, v = rng.standard_normal((2, ny, nx))
        s = fs.GPUFluidSolver(nx=nx, ny=ny, lx=float(nx), ly=float(ny), pressure_solver=solver, pressure_iterations=40,
                              kernel_variant=variant)
        s.upload_velocity(u, v)
        s.run_stage("divergence", 0.01)
        s.run_stage("pressure", 0.01)
        out.append(s.read_field("pressure"))
        s.destroy()
    assert np.array_equal(out[0], out[1])

"""The paired rows of the advection's fast tiles (fs_advect.cu), bit for bit
without a reference: the grid is periodic, so the advection of a rolled field is
the rolled advection, whatever tile, row of a pair or edge a cell falls to.
Against the f64 scheme, and with tiles too fast to be paired (which round the
offsets of a sample differently): test_gpu_parity.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny, nx", [(16, 32), (17, 33), (24, 96), (25, 100), (7, 40), (40, 260), (96, 132)])
@pytest.mark.parametrize("scheme", ["semi-lagrangian", "maccormack"])
@pytest.mark.parametrize("precision", ["f32", "mixed"])
def test_rolled_field(fs, ny, nx, scheme, precision):
    rng = np.random.default_rng(ny * 1000 + nx)
    u, v = rng.uniform(-1.0, 1.0, (2, ny, nx))
    s = fs.GPUFluidSolver(nx=nx, ny=ny, lx=2 * np.pi * nx / ny, ly=2 * np.pi, advection=scheme,
                          pressure_iterations=0, precision=precision)
    dt = 2.5 * 2 * np.pi / ny  # displacements of up to 2.5 cells

    def advect(a, b):
        s.upload_velocity(a, b)
        s.run_stage("advect", dt)
        return [f.reshape(ny, nx) for f in s.read_velocity()]

    ref = advect(u, v)
    assert all(np.isfinite(f).all() for f in ref)
    for roll in ((0, 1), (1, 0), (8, 0), (5, 13), (-3, 31), (9, 64)):
        for f, r in zip(advect(np.roll(u, roll, (0, 1)), np.roll(v, roll, (0, 1))), ref):
            np.testing.assert_array_equal(f, np.roll(r, roll, (0, 1)))
    s.destroy()


def test_two_tiles_per_cta(fs):
    """Large grids stage two tiles a CTA: an odd number of tile rows, edge tiles
    beside inner ones and a last tile cut in both directions, rolled."""
    ny, nx = 2040, 2052
    rng = np.random.default_rng(1)
    u, v = rng.uniform(-1.0, 1.0, (2, ny, nx))
    for scheme in ("semi-lagrangian", "maccormack"):
        s = fs.GPUFluidSolver(nx=nx, ny=ny, lx=2 * np.pi * nx / ny, ly=2 * np.pi, advection=scheme,
                              pressure_iterations=0)
        dt = 2.5 * 2 * np.pi / ny

        def advect(a, b):
            s.upload_velocity(a, b)
            s.run_stage("advect", dt)
            return [f.reshape(ny, nx) for f in s.read_velocity()]

        ref = advect(u, v)
        roll = (17, 41)
        for f, r in zip(advect(np.roll(u, roll, (0, 1)), np.roll(v, roll, (0, 1))), ref):
            np.testing.assert_array_equal(f, np.roll(r, roll, (0, 1)))
        s.destroy()

"""Diffusion made along with the divergence (diffused_faces, fs_pressure.cu)
against the separate passes, bit for bit: one quad a row, quads that wrap, rows
and quads left over in the last block, non-square grids, a batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def steps(fs, ny, nx, variant, **kw):
    rng = np.random.default_rng(ny * 1000 + nx)
    u, v = rng.standard_normal((2, ny * nx))
    s = fs.GPUFluidSolver(nx=nx, ny=ny, nu=1e-2, kernel_variant=variant, **kw)
    s.upload_velocity(u, v)
    s.advance(1e-3, 2)
    out = s.read_velocity()
    s.destroy()
    return out


@pytest.mark.parametrize("ny, nx", [(4, 4), (8, 8), (7, 12), (20, 132), (33, 64), (9, 260)])
@pytest.mark.parametrize("kw", [dict(precision="f32"), dict(precision="mixed")], ids=["f32", "mixed"])
def test_step_equals_separate_passes(fs, ny, nx, kw):
    kw = dict(kw, pressure_solver="jacobi", pressure_iterations=3, lx=float(nx), ly=float(ny))
    for x, y in zip(steps(fs, ny, nx, 0, **kw), steps(fs, ny, nx, 1, **kw)):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("n", [16, 66, 100, 136])
def test_batch_equals_single_solver(fs, n):
    cfg = dict(n=n, nu=1e-2, pressure_solver="multigrid", pressure_iterations=1, precision="mixed", pressure_tol=1e-6,
               max_cycles=60)
    rng = np.random.default_rng(n)
    fields = [rng.standard_normal((2, n * n)) for _ in range(3)]
    batch = fs.GPUFluidBatch([cfg] * 3)
    for m, f in zip(batch.members, fields):
        m.upload_velocity(*f)
    for _ in range(2):
        batch.step(1e-3)
    for m, f in zip(batch.members, fields):
        one = fs.GPUFluidSolver(**cfg)
        one.upload_velocity(*f)
        for _ in range(2):
            one.step(1e-3)
        for x, y in zip(m.read_velocity(), one.read_velocity()):
            assert np.array_equal(x, y)

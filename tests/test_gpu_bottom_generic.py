"""Bottom levels that form none of the compile-time chains (fs_bottom.cu) run the
generic kernel: one doubling of an odd or even coarsest size, coarsest sizes of other
mg_min_size.  Equal bit for bit to the one-kernel-per-pass V-cycle, and in a batch to a
solver alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (cells, mg_min_size): 18 -> 9, ..., 30 -> 15; 64 -> 4; 40 -> 20 below a tile level; 48 alone, and below two
SIZES = [(18, 8), (20, 8), (22, 8), (26, 8), (28, 8), (30, 8), (64, 4), (80, 16), (48, 32), (192, 32)]


def run(fs, n, variant, **kw):
    u, v = np.random.default_rng(n).standard_normal((2, n * n))
    s = fs.GPUFluidSolver(n=n, pressure_solver="multigrid", kernel_variant=variant, **kw)
    s.upload_velocity(u, v)
    s.advance(1e-3, 2)
    out = (s.read_field("pressure"), *s.read_velocity())
    s.destroy()
    return out


@pytest.mark.parametrize("n, smallest", SIZES)
@pytest.mark.parametrize("kw", [
    dict(pressure_iterations=2),
    dict(pressure_iterations=2, precision="mixed", relax=1.2, mg_coarse_sweeps=8),
    dict(pressure_iterations=3, mg_pre_smooth=1, mg_post_smooth=3, mg_coarse_sweeps=1, relax=0.9),
], ids=["f32", "mixed", "f32-1-3"])
def test_generic_equals_one_pass_kernels(fs, n, smallest, kw):
    kw = dict(kw, mg_min_size=smallest)
    for x, y in zip(run(fs, n, 0, **kw), run(fs, n, 1, **kw)):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("n, smallest", [(18, 8), (30, 8), (80, 16)])
def test_generic_in_a_batch(fs, n, smallest):
    cfg = dict(n=n, pressure_solver="multigrid", pressure_iterations=1, precision="mixed", pressure_tol=1e-6,
               max_cycles=60, mg_min_size=smallest)
    b = fs.GPUFluidBatch([cfg] * 2)
    fields = [np.random.default_rng(k).standard_normal((2, n * n)) for k in range(2)]
    for m, f in zip(b.members, fields):
        m.upload_velocity(*f)
    b.step(1e-3)
    for m, f in zip(b.members, fields):
        s = fs.GPUFluidSolver(**cfg)
        s.upload_velocity(*f)
        s.step(1e-3)
        for x, y in zip(m.read_velocity(), s.read_velocity()):
            assert np.array_equal(x, y)
        s.destroy()
    b.destroy()

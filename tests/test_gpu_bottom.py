"""The bottom solve's compile-time level chains (fs_bottom.cu) against the
one-kernel-per-pass V-cycle: equal bit for bit for every coarsest size 8 .. 15,
sweep count and way into the chain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(fs, n, variant, **kw):
    rng = np.random.default_rng(n)
    u, v = rng.standard_normal((2, n * n))
    s = fs.GPUFluidSolver(n=n, pressure_solver="multigrid", kernel_variant=variant, **kw)
    s.upload_velocity(u, v)
    s.run_stage("divergence", 0.01)
    s.run_stage("pressure", 0.01)
    p = s.read_field("pressure")
    s.advance(1e-3, 2)
    out = (p, *s.read_velocity())
    s.destroy()
    return out


@pytest.mark.parametrize("b", range(8, 16))
def test_chain_equals_one_pass_kernels(fs, b):
    sizes = [4 * b, 8 * b] + ([2 * b, b] if b in (8, 12) else [])
    for n in sizes:
        for kw in (dict(pressure_iterations=2), dict(pressure_iterations=2, precision="mixed", relax=1.2,
                                                     mg_coarse_sweeps=8),
                   dict(pressure_iterations=3, mg_pre_smooth=1, mg_post_smooth=3, mg_coarse_sweeps=1, relax=0.9),
                   dict(pressure_iterations=1, mg_pre_smooth=3, mg_post_smooth=1, mg_coarse_sweeps=0)):
            for x, y in zip(run(fs, n, 0, **kw), run(fs, n, 1, **kw)):
                assert np.array_equal(x, y), (n, kw)


@pytest.mark.parametrize("b", [8, 9, 11, 12, 14, 15])
def test_batched_chain_equals_single_solver(fs, b):
    cfg = dict(n=4 * b, pressure_solver="multigrid", pressure_iterations=1, precision="mixed", pressure_tol=1e-6,
               max_cycles=60, relax=1.2)
    batch = fs.GPUFluidBatch([cfg, cfg, dict(cfg, n=8 * b)])
    singles = [fs.GPUFluidSolver(**cfg), fs.GPUFluidSolver(**cfg), fs.GPUFluidSolver(**dict(cfg, n=8 * b))]
    rng = np.random.default_rng(b)
    for m, s in zip(batch.members, singles):
        u, v = rng.standard_normal((2, m.n))
        m.upload_velocity(u, v)
        s.upload_velocity(u, v)
    for _ in range(2):
        batch.step(1e-3)
        for s in singles:
            s.step(1e-3)
    for m, s in zip(batch.members, singles):
        assert m.last_stats()["converged"]
        for x, y in zip(m.read_velocity(), s.read_velocity()):
            assert np.array_equal(x, y)

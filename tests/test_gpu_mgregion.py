"""The multigrid level kernels on register-held regions (fs_mgreg.cuh) against
the one-kernel-per-pass V-cycle, bit for bit: levels smaller than a region,
levels that cut the last region, levels of 2 mod 4 cells (odd coarse level),
every region class, sweep count; the first cycle's own sweep counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(fs, n, variant, side=0, **kw):
    rng = np.random.default_rng(n)
    u, v = rng.standard_normal((2, n * n))
    s = fs.GPUFluidSolver(n=n, pressure_solver="multigrid", kernel_variant=variant, **kw)
    if side:
        s.set_mg_tiles([side] * 16)
    s.upload_velocity(u, v)
    s.advance(1e-3, 2)
    out = (s.read_field("pressure"), *s.read_velocity())
    s.destroy()
    return out


# 66 -> 33, 100 -> 50 and 126 -> 63 have a tile level of 2 mod 4 or 4 mod 8 cells
@pytest.mark.parametrize("n", [66, 72, 100, 126, 132, 200, 264, 504])
@pytest.mark.parametrize("kw", [
    dict(pressure_iterations=2),
    dict(pressure_iterations=2, precision="mixed", relax=1.2),
    dict(pressure_iterations=2, precision="mixed", mg_pre_smooth=1, mg_post_smooth=3),
    dict(pressure_iterations=3, mg_pre_smooth=3, mg_post_smooth=1, relax=0.9),
], ids=["f32", "mixed", "mixed-1-3", "f32-3-1"])
def test_regions_equal_one_pass_kernels(fs, n, kw):
    ref = run(fs, n, 1, **kw)
    for side in (16, 32, 64):
        for x, y in zip(run(fs, n, 0, side, **kw), ref):
            assert np.array_equal(x, y), side


# (the one-pass kernels have no such option)
@pytest.mark.parametrize("first", [(0, 0), (0, 1), (1, 0), (1, 2), (2, 2)])
def test_first_cycle_sweeps(fs, first):
    kw = dict(pressure_iterations=2, precision="mixed")
    for n in (66, 132, 264):
        ref = run(fs, n, 0, 16, mg_first_pre=first[0], mg_first_post=first[1], **kw)
        for side in (32, 64):
            for x, y in zip(run(fs, n, 0, side, mg_first_pre=first[0], mg_first_post=first[1], **kw), ref):
                assert np.array_equal(x, y), (n, side)
        same = all(np.array_equal(x, y) for x, y in zip(run(fs, n, 0, **kw), ref))
        assert same == (first == (2, 2))


@pytest.mark.parametrize("n, count", [(66, 3), (72, 40), (136, 3), (264, 2)])
def test_batch_equals_single_solver(fs, n, count):
    cfg = dict(n=n, pressure_solver="multigrid", pressure_iterations=1, precision="mixed", pressure_tol=1e-6,
               max_cycles=60)
    batch = fs.GPUFluidBatch([cfg] * count)
    rng = np.random.default_rng(n)
    fields = [rng.standard_normal((2, n * n)) for _ in batch.members]
    for m, f in zip(batch.members, fields):
        m.upload_velocity(*f)
    for _ in range(2):
        batch.step(1e-3)
    for k in (0, count - 1):
        one = fs.GPUFluidSolver(**cfg)
        one.upload_velocity(*fields[k])
        for _ in range(2):
            one.step(1e-3)
        for x, y in zip(batch.members[k].read_velocity(), one.read_velocity()):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("precision", ["f32", "mixed"])
def test_level_that_fetches_ahead(fs, precision):
    """Levels of 2896 cells on fetch a later region into L2."""
    kw = dict(pressure_iterations=1, precision=precision)
    for x, y in zip(run(fs, 3072, 0, **kw), run(fs, 3072, 1, **kw)):
        assert np.array_equal(x, y)

"""fs_get_mg_tiles reports the tile sides in use: on a level of 2 mod 4 cells only
side 16 is, whatever is asked for, and the autotuner tries no other there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, used", [
    (66, {32: [16], 64: [16]}),           # 66 -> 33
    (126, {32: [16], 64: [16]}),          # 126 -> 63
    (200, {32: [32, 32], 64: [64, 16]}),  # 200, 100 -> 50
    (264, {32: [32, 32, 16], 64: [64, 64, 16]}),  # 264, 132, 66 -> 33
    (504, {32: [32, 32, 16], 64: [64, 64, 16]}),  # 504, 252, 126 -> 63
])
def test_sides_in_use(fs, n, used):
    s = fs.GPUFluidSolver(n=n, pressure_solver="multigrid", pressure_iterations=2)
    for side, want in used.items():
        s.set_mg_tiles([side] * 16)
        assert s.mg_tiles() == want
    s.set_mg_tiles([])
    u, v = np.random.default_rng(n).standard_normal((2, n * n))
    s.upload_velocity(u, v)
    tuned = s.autotune_tiles(1e-3, 1)["tiles"]
    if used[64][-1] == 16 and used[32][-1] == 16:
        assert tuned[-1] == 16
    s.destroy()


def test_sides_in_use_of_a_batch(fs):
    cfg = dict(n=66, pressure_solver="multigrid", pressure_iterations=1, precision="mixed", pressure_tol=1e-6,
               max_cycles=40)
    b = fs.GPUFluidBatch([cfg] * 4)
    for k, m in enumerate(b.members):
        m.upload_velocity(*np.random.default_rng(k).standard_normal((2, 66 * 66)))
        m.set_mg_tiles([64])
        assert m.mg_tiles() == [16]
    b.autotune_tiles(1e-3, 1)
    for m in b.members:
        assert m.mg_tiles() == [16]
    b.destroy()

"""fs_conv3x3_bf16 takes its biases from any f32 address: a slice that starts
1, 2 or 3 words after a 16-byte boundary gives the same bits as an aligned copy
of it, for every channel pair and epilogue."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

PAIRS = [(16, 16), (16, 32), (32, 16), (32, 64), (64, 32), (64, 128), (128, 64)]


@pytest.mark.parametrize("ci, co, epi", [(a, b, e) for a, b in PAIRS for e in (0, 1)] + [(16, 16, 2), (32, 16, 2)])
def test_bias_at_any_word(fs, ci, co, epi):
    lib = fs._lib.load()
    rng = np.random.default_rng(1000 * ci + 10 * co + epi)
    B, H, W = 1, 9, 37
    x = torch.from_numpy(rng.standard_normal((B, H, W, ci)).astype(np.float32)).cuda().to(torch.bfloat16)
    w = torch.from_numpy(rng.standard_normal((9, ci // 8, co, 8)).astype(np.float32)).cuda().to(torch.bfloat16)
    words = 1 if epi == 2 else co
    bias = rng.standard_normal(words).astype(np.float32)
    outs = []
    for offset in (0, 1, 2, 3):
        room = torch.full((offset + words,), float("nan"), dtype=torch.float32, device="cuda")
        part = room[offset:]
        part.copy_(torch.from_numpy(bias))
        assert part.data_ptr() % 16 == 4 * offset
        out = torch.zeros((B, H, W) if epi == 2 else (B, H, W, co),
                          dtype=torch.float32 if epi == 2 else torch.bfloat16, device="cuda")
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        fs._lib.check(lib.fs_conv3x3_bf16(x.data_ptr(), w.data_ptr(), part.data_ptr(), out.data_ptr(), B, H, W, ci, co,
                                          epi, err.data_ptr(), torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert int(err.item()) == 0
        outs.append(out.float().cpu().numpy())
    assert np.isfinite(outs[0]).all()
    for other in outs[1:]:
        np.testing.assert_array_equal(other, outs[0])

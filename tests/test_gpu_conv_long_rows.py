"""fs_conv3x3_bf16 on an image row of more than 2^31 16-byte pieces (128 channels,
2^27 pixels and more): offsets take 64 bits.  The row repeats every 8 pixels, so the
output does, wherever the pixel lies."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_row_beyond_32_bit_offsets(fs):
    lib = fs._lib.load()
    ci, co, W = 128, 64, 2 ** 27 + 8 * 37
    if torch.cuda.mem_get_info()[0] < 70 * 2 ** 30:
        pytest.skip("needs 52 GB of device memory")
    rng = np.random.default_rng(3)

    def device(a):
        return torch.from_numpy(a.astype(np.float32)).cuda().to(torch.bfloat16)

    period = device(rng.standard_normal((8, ci)))
    w = device(rng.standard_normal((9, ci // 8, co, 8)))
    bias = torch.from_numpy(rng.standard_normal(co).astype(np.float32)).cuda()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def conv(x):
        out = torch.empty((x.shape[0], co), dtype=torch.bfloat16, device="cuda")
        fs._lib.check(lib.fs_conv3x3_bf16(x.data_ptr(), w.data_ptr(), bias.data_ptr(), out.data_ptr(), 1, 1, x.shape[0],
                                          ci, co, 0, err.data_ptr(), torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert int(err.item()) == 0
        return out

    want = conv(period)  # 8 pixels, wrapped
    out = conv(period.repeat(W // 8, 1)).view(W // 8, 8, co)
    for part in (out[:100], out[W // 16 - 50:W // 16 + 50], out[-100:]):
        assert torch.equal(part, want.expand_as(part))
    del out
    torch.cuda.empty_cache()

"""Row kernels in the forms that hold only what a decoder layer's launch runs: bit for bit what the general forms give."""
import pytest
import torch

from util import i32, u8

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4M3 = torch.float8_e4m3fn


# widths: one quad, a ragged last warp, one / two / four quads a thread and the steps between them; rows: one, either side
# of one and of three CTAs an SM
@pytest.mark.parametrize("F", [8, 1032, 4096, 4104, 5120, 5128, 8192, 8200, 13824, 16384])
@pytest.mark.parametrize("M", [1, 148, 149, 444, 445])
def test_gated_quantiser_bits(M, F):
    from instinctflash_b200 import _lib
    from instinctflash_b200.kernels import activation
    lib = _lib.lib()
    g = torch.Generator(device=DEV).manual_seed(M + F)
    dtype = torch.bfloat16 if (M + F // 8) % 2 else torch.float16
    gu = torch.full((M, 2 * F + 8), float("nan"), device=DEV, dtype=dtype)[:, : 2 * F]
    gu.copy_(torch.randn(M, 2 * F, device=DEV, generator=g) * 3)
    gu[M // 2, : F // 2] = 0.0
    gu[M - 1, F - 1], gu[M - 1, F // 2] = float("nan"), float("inf")
    row, col = torch.rand(M, device=DEV, generator=g), torch.rand(2 * F, device=DEV, generator=g)
    for act in (activation.GELU_TANH, activation.SILU):
        for kw in (dict(row=row, col=col), dict(row=row), dict(col=col), {}):
            outs = []
            for group in (0, 256):   # 256: the kernel with a group of 256 threads a row
                q, s = torch.full((M, F + 8), 1.0, device=DEV).to(E4M3), torch.empty(M, device=DEV)
                assert lib.iflb200_row_set_group(group) == 0
                try:
                    activation.gated_act_quant(gu, q[:, :F], s, act=act, **kw)
                finally:
                    assert lib.iflb200_row_set_group(0) == 0
                outs.append((q, s))
            torch.cuda.synchronize()
            assert torch.equal(u8(outs[0][0]), u8(outs[1][0])) and torch.equal(i32(outs[0][1]), i32(outs[1][1]))


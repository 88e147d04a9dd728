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


# A weight of ones takes the general form and multiplies by one.  Widths: quads and chunks with ragged ends, the widest of
# the planes form (2048) and of the bf16 delta's (3072 and beyond); planes: 0 is a bf16 delta, then either side of the groups.
@pytest.mark.parametrize("D", [8, 1016, 1024, 1032, 2048, 2056, 3072, 6152])
@pytest.mark.parametrize("planes", [0, 1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_plain_residual_bits(D, planes, dtype):
    from instinctflash_b200.kernels import norm
    M = 9
    g = torch.Generator(device=DEV).manual_seed(D + planes)
    res0 = (torch.randn(M, D, device=DEV, generator=g) * 2).to(dtype)
    delta = torch.randn(*((planes, M, D) if planes else (M, D)), device=DEV, generator=g)
    if not planes:
        delta = delta.to(torch.bfloat16)
    res0[1], delta[..., 1, :] = 0.0, 0.0                      # nothing: eps alone
    res0[2], delta[..., 2, :] = 1e-25, 0.0                    # squares below the smallest number
    res0[3], delta[..., 3, :] = 1e30, 0.0                     # and above the largest
    res0[4, D // 2], res0[5, D - 1], res0[6, 0] = float("nan"), float("inf"), float("-inf")
    row, col = torch.rand(M, device=DEV, generator=g), torch.rand(D, device=DEV, generator=g)
    for eps in (1e-6, 0.0):
        outs = []
        for weight in (None, torch.ones(D, device=DEV)):
            res, q, s = res0.clone(), torch.full((M, D + 8), 1.0, device=DEV).to(E4M3), torch.empty(M, device=DEV)
            norm.residual_norm_quant(res, delta=delta, delta_row=row, delta_col=col, weight=weight, q=q[:, :D], q_scale=s, eps=eps)
            outs.append((res, q, s))
        torch.cuda.synchronize()
        (r0, q0, s0), (r1, q1, s1) = outs
        assert torch.equal(u8(r0), u8(r1)) and torch.equal(u8(q0), u8(q1)) and torch.equal(i32(s0), i32(s1))


# either side of the 32 MB of planes from which a plain call takes the general form
@pytest.mark.parametrize("M,D,planes", [(512, 2048, 8), (513, 2048, 8), (819, 1280, 8), (820, 1280, 8), (820, 2048, 5)])
def test_plain_residual_bits_of_many_planes(M, D, planes):
    from instinctflash_b200.kernels import norm
    g = torch.Generator(device=DEV).manual_seed(M)
    res0, delta = torch.randn(M, D, device=DEV, generator=g), torch.randn(planes, M, D, device=DEV, generator=g)
    row, col = torch.rand(M, device=DEV, generator=g), torch.rand(D, device=DEV, generator=g)
    outs = []
    for weight in (None, torch.ones(D, device=DEV)):
        res, q, s = res0.clone(), torch.empty(M, D, device=DEV, dtype=E4M3), torch.empty(M, device=DEV)
        norm.residual_norm_quant(res, delta=delta, delta_row=row, delta_col=col, weight=weight, q=q, q_scale=s)
        outs.append((res, q, s))
    torch.cuda.synchronize()
    assert all(torch.equal(u8(a), u8(b)) for a, b in zip(*outs))

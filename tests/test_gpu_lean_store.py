"""The skinny kernel's stores at the edges of its tiles: rows that end in any eight of a quadrant, columns that end in
any sixteen of a tile, K off the 128-byte step.  128-wide tiles of the general kernel give the same bits; guard rows and
columns show that nothing else is written."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4M3 = torch.float8_e4m3fn
ROWS = [1, 8, 9, 16, 17, 50, 63, 64, 65, 80, 81, 97, 127, 128, 129, 300]
COLUMNS = [16, 32, 48, 64, 80, 1040]


def operands(M, N, K):
    from instinctflash_b200.kernels.fp8 import Fp8Weight
    g = torch.Generator(device=DEV).manual_seed(M * 31 + N)
    a, w = torch.randn(M, K, device=DEV, generator=g).to(E4M3), torch.randn(N, K, device=DEV, generator=g).to(E4M3)
    return a, Fp8Weight(w, torch.rand(N, device=DEV, generator=g) + 0.1, torch.randn(N, device=DEV, generator=g)), torch.rand(M, device=DEV, generator=g) + 0.1


def both(run, M, N, dtype):
    """What `run(out)` writes in 64-wide and in 128-wide tiles, guards included; the first is known to have been 64 wide."""
    from instinctflash_b200 import _lib
    lib = _lib.lib()
    outs = []
    try:
        assert lib.iflb200_gemm_set_split_k(1) == 0
        for tile in (64, 128):
            assert lib.iflb200_gemm_set_config(tile, 0, 0) == 0
            out = torch.full((M + 2, N + 16), 7.0, device=DEV, dtype=dtype)
            run(out[:M, :N])
            width = ctypes.c_int(0)
            assert lib.iflb200_gemm_last_launch(None, ctypes.byref(width), None) == 0 and width.value == tile
            outs.append(out)
    finally:
        lib.iflb200_gemm_set_config(0, 0, 0)
        lib.iflb200_gemm_set_split_k(0)
    torch.cuda.synchronize()
    assert (outs[0][M:] == 7.0).all() and (outs[0][:, N:] == 7.0).all()
    assert torch.equal(*[t.view(torch.int32 if dtype == torch.float32 else torch.int16) for t in outs])


@pytest.mark.parametrize("N", COLUMNS)
@pytest.mark.parametrize("M", ROWS)
def test_rows_and_columns(M, N):
    from instinctflash_b200.kernels import fp8
    a, w, s = operands(M, N, 528 if M % 2 else 512)
    both(lambda out: fp8.gemm(a, w, out), M, N, torch.bfloat16)
    for dtype in (torch.bfloat16, torch.float16, torch.float32):
        both(lambda out: fp8.fp8_linear(a, s, w, out), M, N, dtype)
        both(lambda out: fp8.fp8_linear(a, s, w, out, bias=w.bias.to(torch.bfloat16), exact=True), M, N, dtype)
    scalar = fp8.Fp8Weight(w.w, w.scale[:1], None)   # per-tensor scales
    both(lambda out: fp8.fp8_linear(a, s[:1], scalar, out, bias=w.bias, use_weight_bias=False, exact=True), M, N, torch.bfloat16)


@pytest.mark.parametrize("M,N,S", [(1, 16, 3), (9, 80, 2), (50, 1040, 4), (63, 64, 1), (64, 48, 3)])
def test_planes(M, N, S):
    """A plane is the GEMM of its K range: four slabs a stage, ranges in whole stages."""
    from instinctflash_b200.kernels import fp8
    K = 512 * S
    a, w, _ = operands(M, N, K)
    planes = torch.full((S + 1, M, N), 7.0, device=DEV)
    fp8.gemm_partials(a, w, planes[:S])
    for i in range(S):
        k = slice(512 * i, 512 * (i + 1))
        whole = torch.empty(M, N, device=DEV)
        fp8.fp8_linear(a[:, k], None, fp8.Fp8Weight(w.w[:, k], None, None), whole, use_weight_bias=False, exact=True)
        assert torch.equal(planes[i].view(torch.int32), whole.view(torch.int32))
    assert (planes[S] == 7.0).all()

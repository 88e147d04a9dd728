"""The gated GEMM on CTA pairs at the edges of its tiles: rows that end in either CTA of a pair, one block of hidden
units and ragged last ones (16 columns leave as the first half of a store), K off the 128-byte step, several tiles
per pair.  The K loop is that of the single-CTA tiles, so every bit has to be the same."""
import ctypes

import pytest
import torch

from util import i32

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4M3 = torch.float8_e4m3fn


@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("M,F,K", [(1, 128, 16), (128, 144, 80), (129, 272, 512), (257, 400, 1040), (384, 4112, 256), (1000, 16384, 128)])
def test_gated_pairs_equal_single_cta_tiles(M, F, K, act):
    from instinctflash_b200 import _lib
    from instinctflash_b200.kernels import fp8
    lib = _lib.lib()
    g = torch.Generator(device=DEV).manual_seed(M + F + K)
    a = torch.randn(M, K, device=DEV, generator=g).to(E4M3)
    W = fp8.Fp8Weight((torch.randn(2 * F, K, device=DEV, generator=g) * 4).to(E4M3),
                      torch.rand(2 * F, device=DEV, generator=g) * 1e-2, None)
    s = torch.rand(M, device=DEV, generator=g)
    got = []
    try:
        for mode in (1, 3):
            assert lib.iflb200_gemm_set_mode(mode) == 0
            h = torch.full((M + 3, F + 32), float("nan"), device=DEV)
            amax = torch.zeros(M, device=DEV)
            fp8.fp8_linear_gated(a, s, W, h[:M, :F], amax, act=act)
            torch.cuda.synchronize()
            assert torch.equal(amax, h[:M, :F].abs().amax(1))
            got.append(h)
    finally:
        lib.iflb200_gemm_set_mode(0)
    assert torch.equal(i32(got[0]), i32(got[1]))   # guard rows and columns included
    rec = ctypes.c_uint32(0)
    assert lib.iflb200_gemm_take_timeout_record(ctypes.byref(rec), None) == 0 and rec.value == 0

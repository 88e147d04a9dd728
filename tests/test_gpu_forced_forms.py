"""Forced GEMM configurations that do not fit a problem are refused, whatever they are combined with."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4M3 = torch.float8_e4m3fn


# too few K steps for the split, narrower than a CTA pair's tile
@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("M,N,K,split", [(50, 64, 512, 4), (300, 128, 1024, 2)])
def test_a_split_that_does_not_fit_is_refused(mode, M, N, K, split):
    from instinctflash_b200 import _lib
    lib = _lib.lib()
    a, w = (torch.zeros(n, K, device=DEV).to(E4M3) for n in (M, N))
    out = torch.full((M, N), 7.0, device=DEV, dtype=torch.bfloat16)
    try:
        assert lib.iflb200_gemm_set_mode(mode) == 0 and lib.iflb200_gemm_set_split_k(split) == 0
        st = lib.iflb200_gemm_fp8_raw(a.data_ptr(), K, w.data_ptr(), K, M, N, K, out.data_ptr(), N,
                                      torch.cuda.current_stream().cuda_stream)
    finally:
        lib.iflb200_gemm_set_mode(0)
        lib.iflb200_gemm_set_split_k(0)
    torch.cuda.synchronize()
    assert st == _lib.ERR_ARG and (out == 7.0).all()

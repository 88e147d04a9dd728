"""Forced GEMM configurations that do not fit a problem are refused, whatever they are combined with."""
import ctypes

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


# the tokens form has no split over a cluster: asked for together, the split is taken where it fits and refused where not
@pytest.mark.parametrize("M,N,K,split,fits", [(50, 64, 512, 4, False), (300, 128, 1024, 2, False), (300, 256, 4096, 4, True), (301, 2048, 2048, 2, True)])
def test_a_forced_split_stands_above_the_tokens_form(M, N, K, split, fits):
    from instinctflash_b200 import _lib
    lib = _lib.lib()
    g = torch.Generator(device=DEV).manual_seed(K)
    a, w = (torch.randn(n, K, device=DEV, generator=g).to(E4M3) for n in (M, N))
    stream, outs, ran = torch.cuda.current_stream().cuda_stream, [], ctypes.c_int(0)
    try:
        assert lib.iflb200_gemm_set_split_k(split) == 0
        for mode in (128, 256):
            assert lib.iflb200_gemm_set_mode(mode) == 0
            outs.append(torch.full((M, N), 7.0, device=DEV, dtype=torch.bfloat16))
            st = lib.iflb200_gemm_fp8_raw(a.data_ptr(), K, w.data_ptr(), K, M, N, K, outs[-1].data_ptr(), N, stream)
            assert st == (0 if fits else _lib.ERR_ARG)
            assert not fits or (lib.iflb200_gemm_last_launch(None, None, ctypes.byref(ran)) == 0 and ran.value == split)
    finally:
        lib.iflb200_gemm_set_mode(0)
        lib.iflb200_gemm_set_split_k(0)
    torch.cuda.synchronize()
    assert torch.equal(*outs) and bool((outs[0] == 7.0).all()) == (not fits)


# small calls of the fused linear: no K split over a cluster, whose epilogue costs more than the K steps it saves
@pytest.mark.parametrize("M,N,K", [(4, 3408, 7760), (175, 608, 4016), (309, 1840, 5344), (193, 304, 304), (66, 13184, 1248)])
def test_fused_linear_keeps_the_unsplit_bits(M, N, K):
    from instinctflash_b200 import _lib
    from instinctflash_b200.kernels import fp8
    lib = _lib.lib()
    g = torch.Generator(device=DEV).manual_seed(K)
    a = torch.randn(M, K, device=DEV, generator=g).to(E4M3)
    w = fp8.Fp8Weight(torch.randn(N, K, device=DEV, generator=g).to(E4M3), torch.rand(N, device=DEV, generator=g),
                      torch.randn(N, device=DEV, generator=g))
    s = torch.rand(M, device=DEV, generator=g)
    outs = []
    for tile in (0, 64):
        assert lib.iflb200_gemm_set_config(tile, 0, 0) == 0 and lib.iflb200_gemm_set_split_k(1 if tile else 0) == 0
        try:
            y = torch.full((M, N), float("nan"), device=DEV)
            fp8.fp8_linear(a, s, w, y)
            torch.cuda.synchronize()
            outs.append(y)
        finally:
            lib.iflb200_gemm_set_config(0, 0, 0)
            lib.iflb200_gemm_set_split_k(0)
    assert torch.equal(*outs)


# fp32 outputs of the skinny kernel over one row block and several, against the kernel with one K slab a load: last rows in
# each quadrant of a block, columns that end inside a warp's 32, several tiles for a CTA, no scales and all of them
@pytest.mark.parametrize("M,N,K", [(65, 16, 512), (100, 208, 640), (129, 80, 640), (300, 48, 1040), (477, 144, 784), (2100, 720, 512)])
@pytest.mark.parametrize("exact", [False, True])
def test_skinny_fp32_rows(M, N, K, exact):
    from instinctflash_b200 import _lib
    from instinctflash_b200.kernels import fp8
    lib = _lib.lib()
    g = torch.Generator(device=DEV).manual_seed(M)
    a, w = (torch.randn(n, K, device=DEV, generator=g).to(E4M3) for n in (M, N))
    s, c, b = (torch.rand(n, device=DEV, generator=g) for n in (M, N, N))
    outs, tile = [], ctypes.c_int(0)
    try:
        assert lib.iflb200_gemm_set_config(64, 0, 0) == 0 and lib.iflb200_gemm_set_split_k(1) == 0
        for mode in (128, 128 + 4096):
            assert lib.iflb200_gemm_set_mode(mode) == 0
            for row, weight in ((s, fp8.Fp8Weight(w, c, b)), (None, fp8.Fp8Weight(w, None, None))):
                outs.append(torch.full((M + 2, N + 48), float("nan"), device=DEV))
                fp8.fp8_linear(a, row, weight, outs[-1][:M, 16:16 + N], exact=exact)
                assert lib.iflb200_gemm_last_launch(None, ctypes.byref(tile), None) == 0 and tile.value == 64
    finally:
        lib.iflb200_gemm_set_mode(0)
        lib.iflb200_gemm_set_config(0, 0, 0)
        lib.iflb200_gemm_set_split_k(0)
    torch.cuda.synchronize()
    for skinny, general in zip(outs[:2], outs[2:]):
        assert not torch.isnan(skinny[:M, 16:16 + N]).any()
        assert torch.equal(skinny.view(torch.int32), general.view(torch.int32))   # guard rows and columns included

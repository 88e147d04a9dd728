"""The GEMM with tokens on the MMA's N side at the edges of its tiles: one token, tokens that end in either half of a
pair's tile and on either side of a block of 16, weight rows that end in either CTA and inside a warp's 32, an odd
number of K slabs, K off the 128-byte step, several tiles per pair, rings given back one and two slabs at a time.
The K loop is that of the other forms and the epilogues' arithmetic theirs, so every bit has to be the same; guard
rows and columns show that nothing else is written."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4M3 = torch.float8_e4m3fn
# (tokens, columns, K, tile width)
SHAPES = [(1, 16, 16, 64), (17, 256, 384, 64), (64, 272, 128, 64), (97, 528, 1040, 128), (257, 144, 2048, 128), (129, 1024, 640, 192),
          (225, 304, 1152, 224), (333, 2560, 2064, 0), (816, 1040, 512, 256), (301, 2048, 1024, 0), (1000, 4864, 384, 192),
          (5000, 1536, 256, 224)]


def bits(x):
    return x.contiguous().view(torch.int32 if x.dtype == torch.float32 else torch.int16)


def both(run, tile):
    """`run` without the tokens form, then with it; the second is known to have been that form."""
    from instinctflash_b200 import _lib
    lib = _lib.lib()
    out = []
    try:
        assert lib.iflb200_gemm_set_split_k(1) == 0
        for mode in (128, 256):
            assert lib.iflb200_gemm_set_mode(mode) == 0 and lib.iflb200_gemm_set_config(tile if mode == 256 else 0, 0, 0) == 0
            out.append(run())
            fam, width = ctypes.c_int(0), ctypes.c_int(0)
            assert lib.iflb200_gemm_last_launch(ctypes.byref(fam), ctypes.byref(width), None) == 0
            assert bool(fam.value & 4) == (mode == 256) and (mode == 128 or not tile or width.value == tile)
        torch.cuda.synchronize()
    finally:
        lib.iflb200_gemm_set_mode(0)
        lib.iflb200_gemm_set_split_k(0)
        lib.iflb200_gemm_set_config(0, 0, 0)
    rec = ctypes.c_uint32(0)
    assert lib.iflb200_gemm_take_timeout_record(ctypes.byref(rec), None) == 0 and rec.value == 0
    for i, (a, b) in enumerate(zip(*out)):
        assert torch.equal(bits(a), bits(b)), i


def operands(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    a = torch.randn(M, K, device=DEV, generator=g).to(E4M3)
    w = (torch.randn(N, K, device=DEV, generator=g) * 4).to(E4M3)
    return g, a, w


def guarded(M, N, dtype):
    return torch.full((M + 2, N + 48), float("nan"), device=DEV, dtype=dtype)


@pytest.mark.parametrize("M,N,K,tile", SHAPES)
def test_raw_and_dequantised(M, N, K, tile):
    from instinctflash_b200.kernels import fp8
    g, a, w = operands(M, N, K)
    s, t = torch.rand(M, device=DEV, generator=g), torch.rand(1, device=DEV, generator=g)
    c, b = torch.rand(N, device=DEV, generator=g) * 1e-2, torch.randn(N, device=DEV, generator=g)
    W = fp8.Fp8Weight
    scales = [(s, W(w, c, b)), (t, W(w, t, b.bfloat16())), (None, W(w, c, b)), (s, W(w, None, b)), (None, W(w, None, b)), (s, W(w, c, None))]

    def run():
        out = [guarded(M, N, torch.bfloat16)]
        fp8.gemm(a, scales[0][1], out[0][:M, 16:16 + N])
        for dtype in (torch.bfloat16, torch.float16, torch.float32):
            for exact in (False, True):
                for row, weight in scales:
                    out.append(guarded(M, N, dtype))
                    fp8.fp8_linear(a, row, weight, out[-1][:M, 16:16 + N], exact=exact)
        return out
    both(run, tile)


@pytest.mark.parametrize("M,N,K,tile", [s for s in SHAPES if s[2] % 128 == 0])
def test_partial_sums(M, N, K, tile):
    from instinctflash_b200.kernels import fp8
    _, a, w = operands(M, N, K)

    def run():
        out = [torch.full((S + 1, M, N), float("nan"), device=DEV) for S in (1, 2, 3) if S <= (K // 128 + 3) // 4]
        for o in out:
            fp8.gemm_partials(a, fp8.Fp8Weight(w, None, None), o[:-1])
        return out
    both(run, tile)


@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("M,N,K,tile", [s for s in SHAPES if s[1] % 32 == 0])
def test_gated(M, N, K, tile, act):
    from instinctflash_b200.kernels import fp8
    g, a, w = operands(M, N, K)
    F = N // 2
    s, W = torch.rand(M, device=DEV, generator=g), fp8.Fp8Weight(w, torch.rand(N, device=DEV, generator=g) * 1e-2, None)

    def run():
        h, amax = torch.full((M + 3, F + 32), float("nan"), device=DEV), torch.zeros(M + 1, device=DEV)
        fp8.fp8_linear_gated(a, s, W, h[:M, :F], amax[:M], act=act)
        assert torch.equal(amax[:M], h[:M, :F].abs().amax(1))
        return [h, amax]
    both(run, tile)


# Reductions that are split over a cluster without the form, over sizes at which it is estimated faster unsplit; the last
# rows on both sides of K = 14336
@pytest.mark.parametrize("M,N,K", [(71, 304, 4864), (166, 1232, 5184), (411, 2112, 8896), (510, 320, 9296), (260, 3072, 13824),
                                   (260, 3072, 14208), (260, 3072, 14336), (260, 3072, 16384)])
def test_the_choice_keeps_the_k_split(M, N, K):
    from instinctflash_b200 import _lib
    from instinctflash_b200.kernels import fp8
    lib = _lib.lib()
    g, a, w = operands(M, N, K)
    s = torch.rand(M, device=DEV, generator=g)
    W = fp8.Fp8Weight(w, torch.rand(N, device=DEV, generator=g) * 1e-2, torch.randn(N, device=DEV, generator=g))
    calls = [lambda o: fp8.gemm(a, W, o), lambda o: fp8.fp8_linear(a, s, W, o), lambda o: fp8.fp8_linear(a, s, W, o, exact=True)]
    outs, splits = [], []
    try:
        for mode in (128, 0):
            assert lib.iflb200_gemm_set_mode(mode) == 0
            for call in calls:
                outs.append(torch.full((M, N), float("nan"), device=DEV, dtype=torch.bfloat16))
                call(outs[-1])
                split = ctypes.c_int(0)
                assert lib.iflb200_gemm_last_launch(None, None, ctypes.byref(split)) == 0
                splits.append(split.value)
    finally:
        lib.iflb200_gemm_set_mode(0)
    assert splits[:3] == splits[3:] and max(splits) > 1
    for without, default in zip(outs[:3], outs[3:]):
        assert torch.equal(bits(without), bits(default))


# more than 1500 rows: few columns stay with the 64-wide form, up to 512 of them; the sizes around the line keep theirs
@pytest.mark.parametrize("M,N,K,taken", [(6808, 32, 2224, False), (2588, 288, 3984, False), (4394, 16, 3456, False), (1500, 80, 6560, True),
                                         (1650, 704, 1376, True), (7032, 416, 4416, True)])
def test_few_columns_of_many_rows(M, N, K, taken):
    from instinctflash_b200 import _lib
    from instinctflash_b200.kernels import fp8
    g, a, w = operands(M, N, K)
    s, W = torch.rand(M, device=DEV, generator=g), fp8.Fp8Weight(w, torch.rand(N, device=DEV, generator=g), None)
    family = ctypes.c_int(0)
    for call in (lambda o: fp8.gemm(a, W, o), lambda o: fp8.fp8_linear(a, s, W, o)):
        call(torch.empty(M, N, device=DEV, dtype=torch.bfloat16))
        assert _lib.lib().iflb200_gemm_last_launch(ctypes.byref(family), None, None) == 0
        assert bool(family.value & 4) == taken

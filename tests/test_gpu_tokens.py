"""The GEMM with tokens on the MMA's N side at the edges of its tiles: one token, tokens that end in either half of a
pair's tile and on either side of a block of 16, weight rows that end in either CTA and inside a warp's 32, an odd
number of K slabs, K off the 128-byte step, rings given back one and two slabs at a time, each with more tiles than two
a pair (accumulators given back, ring phases carried over) and slab counts that wrap the ring inside a tile.
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
          (5000, 1536, 256, 224),
          # two slabs at a time: three tiles and more for a pair, an odd and an even number of slabs; K ranges of four and five slabs in turn
          (1000, 4864, 384, 64), (1000, 4864, 1152, 128), (1000, 4864, 1024, 64), (1000, 1536, 1664, 64)]
# Widths of the choice that no setting names, at sizes that it gives them: 96, 144 and 160 on either side of the line
# between the two rings, 48 and 240 at the ends.  (width, tokens, columns, K, K ranges)
RAW_WIDTHS = [(48, 66, 256, 640, 1), (96, 163, 6208, 640, 1), (144, 1515, 256, 640, 1), (160, 1035, 7456, 640, 1), (240, 1348, 7968, 640, 1)]
DEQUANT_WIDTHS = [(48, 66, 256, 640, 1), (96, 324, 3104, 640, 1), (144, 1515, 256, 640, 1), (160, 1058, 7456, 640, 1), (240, 1677, 6304, 640, 1)]
PLANES_WIDTHS = [(48, 66, 256, 640, 2), (96, 81, 4672, 640, 2), (144, 258, 6240, 1152, 3), (160, 289, 6176, 1152, 3), (240, 681, 6944, 640, 2)]
GATED_WIDTHS = [(48, 66, 256, 640, 1), (96, 641, 7456, 1424, 1), (144, 970, 7488, 784, 1), (160, 1035, 7456, 640, 1), (240, 1348, 7968, 640, 1)]


def bits(x):
    return x.contiguous().view(torch.int32 if x.dtype == torch.float32 else torch.int16)


def both(run, tile, chosen=0):
    """`run` without the tokens form, then with it; the second is known to have been that form, in tiles of `tile` tokens
    where that is set and of `chosen` where that is expected of the choice."""
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
            assert bool(fam.value & 4) == (mode == 256) and (mode == 128 or not (tile or chosen) or width.value == (tile or chosen))
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


def raw_call(a, w, chosen=0, tile=0):
    from instinctflash_b200.kernels import fp8
    M, N = a.shape[0], w.shape[0]

    def run():
        out = guarded(M, N, torch.bfloat16)
        fp8.gemm(a, fp8.Fp8Weight(w, None, None), out[:M, 16:16 + N])
        return [out]
    both(run, tile, chosen)


def linear_call(g, a, w, chosen=0, tile=0):
    from instinctflash_b200.kernels import fp8
    M, N = a.shape[0], w.shape[0]
    s, t = torch.rand(M, device=DEV, generator=g), torch.rand(1, device=DEV, generator=g)
    c, b = torch.rand(N, device=DEV, generator=g) * 1e-2, torch.randn(N, device=DEV, generator=g)
    W = fp8.Fp8Weight
    scales = [(s, W(w, c, b)), (t, W(w, t, b.bfloat16())), (None, W(w, c, b)), (s, W(w, None, b)), (None, W(w, None, b)), (s, W(w, c, None))]

    def run():
        out = []
        for dtype in (torch.bfloat16, torch.float16, torch.float32):
            for exact in (False, True):
                for row, weight in scales:
                    out.append(guarded(M, N, dtype))
                    fp8.fp8_linear(a, row, weight, out[-1][:M, 16:16 + N], exact=exact)
        return out
    both(run, tile, chosen)


def planes_call(a, w, ranges, chosen=0, tile=0):
    from instinctflash_b200.kernels import fp8

    def run():
        out = [torch.full((S + 1, a.shape[0], w.shape[0]), float("nan"), device=DEV) for S in ranges]
        for o in out:
            fp8.gemm_partials(a, fp8.Fp8Weight(w, None, None), o[:-1])
        return out
    both(run, tile, chosen)


def gated_call(g, a, w, act, chosen=0, tile=0, finite=True):
    from instinctflash_b200.kernels import fp8
    M, N = a.shape[0], w.shape[0]
    F = N // 2
    s, W = torch.rand(M, device=DEV, generator=g), fp8.Fp8Weight(w, torch.rand(N, device=DEV, generator=g) * 1e-2, None)

    def run():
        h, amax = torch.full((M + 3, F + 32), float("nan"), device=DEV), torch.zeros(M + 1, device=DEV)
        fp8.fp8_linear_gated(a, s, W, h[:M, :F], amax[:M], act=act)
        assert not finite or torch.equal(amax[:M], h[:M, :F].abs().amax(1))
        return [h, amax]
    both(run, tile, chosen)


@pytest.mark.parametrize("M,N,K,tile", SHAPES)
def test_raw_and_dequantised(M, N, K, tile):
    g, a, w = operands(M, N, K)
    raw_call(a, w, tile=tile)
    linear_call(g, a, w, tile=tile)


@pytest.mark.parametrize("M,N,K,tile", [s for s in SHAPES if s[2] % 128 == 0])
def test_partial_sums(M, N, K, tile):
    _, a, w = operands(M, N, K)
    planes_call(a, w, [S for S in (1, 2, 3) if S <= (K // 128 + 3) // 4], tile=tile)


@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("M,N,K,tile", [s for s in SHAPES if s[1] % 32 == 0])
def test_gated(M, N, K, tile, act):
    g, a, w = operands(M, N, K)
    gated_call(g, a, w, act, tile=tile)


@pytest.mark.parametrize("form,sizes", [(f, s) for f, t in (("raw", RAW_WIDTHS), ("linear", DEQUANT_WIDTHS), ("planes", PLANES_WIDTHS),
                                                            ("gated", GATED_WIDTHS)) for s in t])
def test_widths_of_the_choice(form, sizes):
    width, M, N, K, S = sizes
    g, a, w = operands(M, N, K)
    if form == "raw":
        raw_call(a, w, chosen=width)
    elif form == "linear":
        linear_call(g, a, w, chosen=width)
    elif form == "planes":
        planes_call(a, w, [S], chosen=width)
    else:
        gated_call(g, a, w, 1, chosen=width)


# codes of NaN in a token and in a weight row, sums that overflow f16
@pytest.mark.parametrize("M,N,K,tile", [(97, 544, 1040, 128), (225, 320, 1152, 224)])
def test_codes_that_are_not_numbers(M, N, K, tile):
    g, a, w = operands(M, N, K)
    a.view(torch.uint8)[5, 7] = 0x7F
    w.view(torch.uint8)[N - 3, K - 1] = 0xFF
    a[M - 1], w[:8] = 448.0, 448.0
    raw_call(a, w, tile=tile)
    linear_call(g, a, w, tile=tile)
    if K % 128 == 0:
        planes_call(a, w, [1, 2], tile=tile)
    gated_call(g, a, w, 0, tile=tile, finite=False)
    gated_call(g, a, w, 1, tile=tile, finite=False)


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


# raw outputs of five K steps and fewer in more than one wave stay with the 256-wide form, six steps and one wave do not
@pytest.mark.parametrize("M,N,K,taken", [(2967, 14016, 384, False), (5117, 7424, 640, False), (3732, 10016, 768, True), (1222, 3552, 512, True)])
def test_short_raw_reductions(M, N, K, taken):
    from instinctflash_b200 import _lib
    from instinctflash_b200.kernels import fp8
    _, a, w = operands(M, N, K)
    fp8.gemm(a, fp8.Fp8Weight(w, None, None), torch.empty(M, N, device=DEV, dtype=torch.bfloat16))
    family = ctypes.c_int(0)
    assert _lib.lib().iflb200_gemm_last_launch(ctypes.byref(family), None, None) == 0
    assert bool(family.value & 4) == taken


@pytest.mark.parametrize("M,N,taken", [(19882, 32, False), (1501, 64, False), (1500, 64, True), (1501, 80, True), (65, 16, True)])
def test_planes_of_few_columns(M, N, taken):
    from instinctflash_b200 import _lib
    from instinctflash_b200.kernels import fp8
    _, a, w = operands(M, N, 2688)
    out = torch.full((6, M, N), float("nan"), device=DEV)
    fp8.gemm_partials(a, fp8.Fp8Weight(w, None, None), out[:5])
    family = ctypes.c_int(0)
    assert _lib.lib().iflb200_gemm_last_launch(ctypes.byref(family), None, None) == 0
    assert bool(family.value & 4) == taken and family.value & 16
    # row 5 * M of the planes is the guard's first; 21 slabs in five ranges of whole stages of four
    assert torch.isnan(out[5]).all()
    cuts = [512 * (6 * i // 5) for i in range(5)] + [2688]
    for i in range(5):
        want = a[:70, cuts[i]:cuts[i + 1]].double() @ w[:, cuts[i]:cuts[i + 1]].double().T
        assert (out[i, :70].double() - want).norm() < 1e-5 * want.norm()
    torch.cuda.synchronize()

"""A weight packed by the kernel directly before a GEMM of more than 2048 rows: such a GEMM reads its weights behind that
kernel, in every form, eagerly and in a captured graph."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4M3 = torch.float8_e4m3fn
N, K = 2048, 2048

# (form, mode, tile): the choice's own, single CTAs, pairs with one and two accumulators, tokens, skinny
FORMS = [("raw", 0, 0), ("raw", 1, 128), ("raw", 2, 0), ("raw", 3, 0), ("raw", 256, 0), ("raw", 1, 64), ("linear", 0, 0),
         ("linear", 256, 128), ("planes", 0, 0), ("gated", 0, 0), ("gated", 128, 0), ("residual", 0, 0)]


@pytest.mark.parametrize("form,mode,tile", FORMS)
@pytest.mark.parametrize("M", [2049, 4680])
def test_weight_packed_directly_before(M, form, mode, tile):
    from instinctflash_b200 import _lib
    from instinctflash_b200.kernels import fp8, norm
    lib = _lib.lib()
    g = torch.Generator(device=DEV).manual_seed(M)
    src = torch.randn(N, K, device=DEV, generator=g).to(torch.bfloat16)
    w = fp8.Fp8Weight(torch.zeros(N, K, device=DEV).to(E4M3), torch.zeros(N, device=DEV), None)
    a, s = torch.randn(M, K, device=DEV, generator=g).to(E4M3), torch.rand(M, device=DEV, generator=g)
    out = {"raw": lambda: torch.zeros(M, N, device=DEV, dtype=torch.bfloat16), "planes": lambda: torch.zeros(2, M, N, device=DEV),
           "linear": lambda: torch.zeros(M, N, device=DEV, dtype=torch.bfloat16), "gated": lambda: torch.zeros(M, N // 2, device=DEV),
           "residual": lambda: torch.zeros(M, N, device=DEV)}[form]()
    amax = torch.zeros(M, device=DEV)

    def gemm():
        if form == "raw":
            fp8.gemm(a, w, out)
        elif form == "linear":
            fp8.fp8_linear(a, s, w, out)
        elif form == "planes":
            fp8.gemm_partials(a, w, out)
        elif form == "gated":
            fp8.fp8_linear_gated(a, s, w, out, amax)
        else:
            fp8.fp8_linear_residual(a, s, w, out)

    def chain(sync=lambda: None):
        norm.row_quant(src, w.w, w.scale)
        sync()
        gemm()
        sync()

    def clear():   # what a GEMM that starts too early would read
        w.w.view(torch.uint8).zero_()
        out.zero_()
        amax.zero_()
        torch.cuda.synchronize()

    try:
        assert lib.iflb200_gemm_set_mode(mode) == 0 and lib.iflb200_gemm_set_config(tile, 0, 0) == 0
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            chain()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            chain()
        for launch in (graph.replay, chain, graph.replay):
            src.copy_(torch.randn(N, K, device=DEV, generator=g))
            clear()
            chain(torch.cuda.synchronize)
            want = out.clone()
            clear()
            launch()
            torch.cuda.synchronize()
            assert torch.equal(out, want) and want.any()
    finally:
        lib.iflb200_gemm_set_mode(0)
        lib.iflb200_gemm_set_config(0, 0, 0)

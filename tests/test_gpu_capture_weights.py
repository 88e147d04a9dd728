"""Weights packed inside a captured graph: a GEMM may start on its weights before the kernel in front of it
has finished, so the kernels in between must not let it start while the packing kernel still writes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4M3 = torch.float8_e4m3fn


# what lies between the packing of the weight and the GEMM that reads it: r = a row kernel, g = another GEMM
@pytest.mark.parametrize("between", ["r", "rr", "rrrr", "gr", "rgr", "g", "grr"])
@pytest.mark.parametrize("ahead", [False, True])
def test_weight_packed_in_the_graph(between, ahead):
    from instinctflash_b200.kernels import fp8, norm
    g = torch.Generator(device=DEV).manual_seed(len(between))
    M, N, K = 50, 2048, 2048
    src = torch.randn(N, K, device=DEV, generator=g).to(torch.bfloat16)
    w = fp8.Fp8Weight(torch.zeros(N, K, device=DEV).to(E4M3), torch.zeros(N, device=DEV), None)
    other = fp8.quantize_weight(torch.randn(1024, 1024, device=DEV, generator=g))
    x, small = (torch.randn(M, n, device=DEV, generator=g).to(torch.bfloat16) for n in (K, 1024))
    xq, sq = (torch.zeros_like(t).to(E4M3) for t in (x, small))
    xs, ss = torch.zeros(M, device=DEV), torch.zeros(M, device=DEV)
    raw, out = torch.zeros(M, 1024, device=DEV, dtype=torch.bfloat16), torch.zeros(M, N, device=DEV, dtype=torch.bfloat16)

    def chain(sync=lambda: None):
        if ahead:   # the packing kernel itself follows a GEMM
            fp8.gemm(sq, other, raw)
        sync()
        norm.row_quant(src, w.w, w.scale)
        sync()
        for what in between:
            fp8.gemm(sq, other, raw) if what == "g" else norm.row_quant(small, sq, ss)
            sync()
        fp8.gemm(xq, w, out)
        sync()

    norm.row_quant(x, xq, xs)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        chain()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain()
    for _ in range(6):
        src.copy_(torch.randn(N, K, device=DEV, generator=g))
        chain(torch.cuda.synchronize)
        want = out.clone()
        w.w.view(torch.uint8).zero_()   # what a GEMM that starts too early would read
        out.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)

"""Calls of thousands of rows are launched dependently too: a stack of diffusion blocks and calls one behind the other give the
bits of plain stream order, with inputs that change from pass to pass."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4M3 = torch.float8_e4m3fn


@pytest.fixture(params=[1, 0], ids=["dependent", "plain"])
def mode(request):
    from instinctflash_b200 import _lib
    lib = _lib.lib()
    assert lib.iflb200_set_dependent_launch(request.param) == 0
    yield request.param
    assert lib.iflb200_set_dependent_launch(1) == 0


results = {}


@pytest.mark.parametrize("M", [2049, 3001])
def test_rows_beyond_two_thousand(M, mode):
    from instinctflash_b200 import stack
    from instinctflash_b200.kernels import fp8, norm
    from instinctflash_b200.runtime.fp8_pack import dynamic_pack_bf16_e4m3
    spec = stack.StackSpec("rows", "wan", 2, M, 1536, 2048, 4608, o_in=1536, cross=True, seed=11)
    weights = stack.make_weights(spec, DEV)
    x, attn = stack.make_inputs(spec, DEV)
    st = stack.LinearStack(spec, weights, DEV)
    st.load(x, attn)
    graph = st.capture()
    outs = []
    w = fp8.quantize_weight(torch.randn(1024, 1536, device=DEV, generator=torch.Generator(device=DEV).manual_seed(3)))
    q, s, y = torch.empty(M, 1536, device=DEV, dtype=E4M3), torch.empty(M, device=DEV), torch.empty(M, 1024, device=DEV, dtype=torch.bfloat16)
    for i in range(4):
        st.load(x * (i + 1), attn)
        graph.replay()
        norm.row_quant(st.res, q, s)          # behind the graph, in the eager stream
        fp8.fp8_linear(q, s, w, y)
        p, scale = dynamic_pack_bf16_e4m3(y)
        outs += [st.res.clone(), y.clone(), p.view(torch.uint8).clone(), scale.clone()]
    torch.cuda.synchronize()
    if mode == 1:
        results[M] = outs
    else:
        assert all(torch.equal(a, b) for a, b in zip(results[M], outs))

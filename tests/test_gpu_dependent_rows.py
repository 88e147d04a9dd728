"""Calls of thousands of rows give the bits of plain stream order, whichever of them are launched dependently: stacks, and
kernels directly behind the kernel that writes their input, with inputs that change from pass to pass."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4M3 = torch.float8_e4m3fn
BF16 = torch.bfloat16


def same_in_every_mode(run):
    """``run`` returns tensors; the dependent modes (1: by size, 2: always) give those of plain order."""
    from instinctflash_b200 import _lib
    lib, want = _lib.lib(), None
    try:
        for mode in (0, 1, 2):
            assert lib.iflb200_set_dependent_launch(mode) == 0
            outs = run()
            torch.cuda.synchronize()
            outs = [t.contiguous().view(torch.uint8) for t in outs]
            assert want is None or all(torch.equal(a, b) for a, b in zip(want, outs)), mode
            want = want or outs
    finally:
        lib.iflb200_set_dependent_launch(1)


def randn(*shape, seed=0):
    return torch.randn(*shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed))


@pytest.mark.parametrize("M", [2049, 3001])
def test_rows_beyond_two_thousand(M):
    from instinctflash_b200 import stack
    from instinctflash_b200.kernels import fp8, norm
    from instinctflash_b200.runtime.fp8_pack import dynamic_pack_bf16_e4m3
    spec = stack.StackSpec("rows", "wan", 2, M, 1536, 2048, 4608, o_in=1536, cross=True, seed=11)
    weights = stack.make_weights(spec, DEV)
    x, attn = stack.make_inputs(spec, DEV)
    w = fp8.quantize_weight(randn(1024, 1536, seed=3))

    def run():
        st = stack.LinearStack(spec, weights, DEV)
        st.load(x, attn)
        graph = st.capture()
        q, s, y = torch.empty(M, 1536, device=DEV, dtype=E4M3), torch.empty(M, device=DEV), torch.empty(M, 1024, device=DEV, dtype=BF16)
        outs = []
        for i in range(4):
            st.load(x * (i + 1), attn)
            graph.replay()
            norm.row_quant(st.res, q, s)          # behind the graph, in the eager stream
            fp8.fp8_linear(q, s, w, y)
            p, scale = dynamic_pack_bf16_e4m3(y)
            outs += [st.res.clone(), y.clone(), p.clone(), scale.clone()]
        return outs

    same_in_every_mode(run)


# gated GEMM, quantiser from its maxima and the two buffers of them in turn; row kernel instead; planes for down
@pytest.mark.parametrize("M,ffn,fused", [(2049, 1024, True), (3000, 4096, True), (2049, 1024, False), (3000, 2048, False)])
def test_decoder_layers_beyond_two_thousand(M, ffn, fused):
    from instinctflash_b200 import stack
    spec = stack.StackSpec("rows", "gemma", 3, M, 1024, ffn, 1536, o_in=1024, seed=5)
    weights = stack.make_weights(spec, DEV)
    x, attn = stack.make_inputs(spec, DEV)

    def run():
        st = stack.LinearStack(spec, weights, DEV, fused=fused)
        st.load(x, attn)
        graph = st.capture()
        outs = []
        for i in range(4):
            st.load(x * (i + 1), attn)
            graph.replay()
            outs.append(st.res.clone())
        return outs

    same_in_every_mode(run)


@pytest.mark.parametrize("M", [2049, 3500])
def test_consumers_directly_behind_their_producer(M):
    from instinctflash_b200.kernels import activation, attention, fp8, norm, rope, wan
    HQ, HKV, HD = 12, 4, 64
    width, D = (HQ + 2 * HKV) * HD, 1536
    w = {n: fp8.quantize_weight(randn(n, 1024, seed=n)) for n in (width, 3 * D, 2 * HQ * HD)}
    inv = rope.rope_inv_freq(HD, 10000.0, DEV)
    pos = torch.arange(M, device=DEV).float()[:, None].contiguous()
    pos3, sections, inv3 = pos.expand(M, 3).contiguous(), (torch.arange(64, device=DEV) % 3).int(), rope.rope_inv_freq(128, 10000.0, DEV)

    def run():
        outs = []
        a, s = torch.empty(M, 1024, device=DEV, dtype=E4M3), torch.empty(M, device=DEV)
        raw = {n: torch.zeros(M, n, device=DEV, dtype=BF16) for n in w}
        q, k = torch.zeros(M, HQ, HD, device=DEV, dtype=BF16), torch.zeros(M, HKV, HD, device=DEV, dtype=BF16)
        v, wq = k.clone(), torch.zeros(M, D, device=DEV, dtype=BF16)
        wk = torch.zeros(1, M, D, device=DEV, dtype=BF16)
        wv = wk.clone()
        q8, qs = torch.zeros(M, HQ * HD, device=DEV).to(E4M3), torch.zeros(M, device=DEV)
        g8, d = torch.zeros_like(q8), torch.zeros(M, HQ * HD, device=DEV)
        ws = attention.SplitWorkspace(1, M, HQ, HKV, HD, 2, DEV)
        ws.po.zero_(), ws.pm.zero_(), ws.pl.fill_(1.0)
        po = ws.po[: M * HQ * HD].view(M, HQ * HD)   # the first of two key ranges
        for i in range(3):
            norm.row_quant(randn(M, 1024, seed=i).to(BF16), a, s)
            fp8.gemm(a, w[width], raw[width])
            rope.qkv_split(raw[width], q, k, v, heads_q=HQ, heads_kv=HKV, head_dim=HD, row=s, inv_freq=inv, pos=pos)
            fp8.gemm(a, w[3 * D], raw[3 * D])
            wan.wan_qkv(raw[3 * D], wq, heads=12, head_dim=128, tokens=M, k_pool=wk, v_pool=wv, row=s, col=w[3 * D].scale, pos=pos3,
                        sections=sections, inv_freq=inv3)
            fp8.gemm(a, w[2 * HQ * HD], raw[2 * HQ * HD])
            activation.gated_act_quant(raw[2 * HQ * HD], g8, qs, row=s)
            norm.dequant_rows(raw[2 * HQ * HD][:, : HQ * HD], po)
            attention.attn_combine(ws, q8=q8, q8_scale=qs, heads_q=HQ, heads_kv=HKV, head_dim=HD, tokens=M)
            norm.dequant_rows(raw[2 * HQ * HD][:, HQ * HD:], d)
            outs += [t.clone() for t in (q, k, v, wq, wk, wv, g8, q8, qs, d)]
        return outs

    same_in_every_mode(run)

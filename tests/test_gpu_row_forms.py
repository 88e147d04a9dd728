"""Row operators on either side of the lines where another form of the kernel takes over: a row's bits do not depend
on how many rows it comes with."""
import pytest
import torch

from util import i32, u8

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4M3 = torch.float8_e4m3fn


# pieces of 1024, 2048 and 4096 columns, each with a ragged last one; the lines are 888 pieces and 2^21 elements
@pytest.mark.parametrize("M,F", [(888, 1024), (444, 1032), (445, 1032), (889, 1024), (222, 4096), (223, 4096), (130, 6152), (511, 4104), (512, 4104),
                                 (2040, 1040), (2050, 1040)])
def test_quantiser_pass_from_known_maxima(M, F):
    from instinctflash_b200.kernels import norm
    g = torch.Generator(device=DEV).manual_seed(M + F)
    h = torch.randn(M, F, device=DEV, generator=g)
    amax, zero = h.abs().amax(1), torch.full((M,), 3.0, device=DEV)
    q, s = torch.full((M, F + 8), 1.0, device=DEV).to(E4M3), torch.empty(M, device=DEV)
    norm.quant_from_amax(h, amax, q[:, :F], s, zero=zero)
    q2, s2, a2 = torch.empty(M, F, device=DEV, dtype=E4M3), torch.empty(M, device=DEV), amax.clone()
    norm.row_quant_from_amax(h, a2, q2, s2)   # one CTA per row
    torch.cuda.synchronize()
    assert torch.equal(u8(q[:, :F]), u8(q2)) and torch.equal(i32(s), i32(s2))
    assert (q[:, F:].float() == 1.0).all() and (zero == 0).all() and torch.equal(amax, h.abs().amax(1))


@pytest.mark.parametrize("hq,hkv,hd", [(8, 1, 256), (8, 8, 64), (16, 2, 128), (16, 1, 256)])
@pytest.mark.parametrize("splits", [3, 8, 13])
@pytest.mark.parametrize("tokens", [148, 149, 296, 297])
def test_merge_does_not_depend_on_the_tokens(tokens, hq, hkv, hd, splits):
    from instinctflash_b200.kernels import attention
    g = torch.Generator(device=DEV).manual_seed(tokens + splits)
    ws = attention.SplitWorkspace(1, tokens, hq, hkv, hd, splits, DEV)
    ws.po.normal_(generator=g)
    ws.pm.normal_(generator=g)
    ws.pl.uniform_(1.0, 50.0, generator=g)
    kw = dict(heads_q=hq, heads_kv=hkv, head_dim=hd)

    def merge(w, n):
        q, s = torch.empty(n, hq * hd, device=DEV, dtype=E4M3), torch.empty(n, device=DEV)
        attention.attn_combine(w, tokens=n, q8=q, q8_scale=s, **kw)
        return q, s

    q, s = merge(ws, tokens)
    for lo in (0, tokens - 5):   # five tokens by themselves: partials are [split][kv head][token * group]
        few = attention.SplitWorkspace(1, 5, hq, hkv, hd, splits, DEV)
        for name, width in (("po", few.po.numel() // few.pm.numel()), ("pm", 1), ("pl", 1)):
            rows = getattr(ws, name)[: splits * tokens * hq * width].view(splits, hkv, tokens, -1)
            getattr(few, name).copy_(rows[:, :, lo:lo + 5].reshape(-1))
        q5, s5 = merge(few, 5)
        torch.cuda.synchronize()
        assert torch.equal(u8(q[lo:lo + 5]), u8(q5)) and torch.equal(i32(s[lo:lo + 5]), i32(s5))


@pytest.mark.parametrize("T,HQ,HKV,HD", [(1199, 16, 2, 256), (1200, 16, 2, 256), (1699, 8, 1, 256), (1700, 8, 1, 256), (370, 14, 1, 256), (371, 14, 1, 256),
                                         (1700, 8, 1, 128), (1699, 8, 1, 128), (1500, 5, 1, 64), (296, 12, 1, 64)])
def test_qkv_rows_do_not_depend_on_the_tokens(T, HQ, HKV, HD):
    from instinctflash_b200.kernels import rope
    g = torch.Generator(device=DEV).manual_seed(T)
    W = (HQ + 2 * HKV) * HD
    raw = torch.randn(T, W, device=DEV, generator=g).to(torch.bfloat16)
    row, pos = torch.rand(T, device=DEV, generator=g), (torch.rand(T, 1, device=DEV, generator=g) * 900).floor()
    kw = dict(heads_q=HQ, heads_kv=HKV, head_dim=HD, col=torch.rand(W, device=DEV, generator=g), bias=torch.randn(W, device=DEV, generator=g),
              inv_freq=rope.rope_inv_freq(HD, 10000.0, DEV))

    def outs():
        return [torch.full((T + 1, h, HD), 7.0, device=DEV, dtype=torch.float16) for h in (HQ, HKV, HKV)]

    whole, pieces = outs(), outs()
    rope.qkv_split(raw, *whole, row=row, pos=pos, **kw)
    for lo in range(0, T, 200):   # calls of 200 tokens: a warp per token and head
        hi = min(T, lo + 200)
        rope.qkv_split(raw[lo:hi], *[t[lo:hi] for t in pieces], row=row[lo:hi], pos=pos[lo:hi], **kw)
    torch.cuda.synchronize()
    for a, b in zip(whole, pieces):
        assert torch.equal(a, b) and (a[T] == 7.0).all()

"""The row kernels for many rows: same codes as the one-row-per-group kernels (GELU quantiser), the
oracle's values (residual + layer norm + quantiser) at the edges of their range."""
import pytest
import torch

from util import assert_quant_close_to_oracle, code_steps, i32, u8

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4M3 = torch.float8_e4m3fn


@pytest.fixture(scope="module")
def lib():
    from instinctflash_b200 import _lib
    return _lib.lib()


def narrow(lib, call):
    """``call`` on the kernels that give each row a group of 256 threads."""
    assert lib.iflb200_row_set_group(256) == 0
    try:
        call()
        torch.cuda.synchronize()
    finally:
        assert lib.iflb200_row_set_group(0) == 0


# widths: smallest, not a whole number of chunks per thread, two groups of 448, the widest; rows: fewer than
# two turns, a last turn with one row, several turns
@pytest.mark.parametrize("M,K,dtype,bias", [(2100, 1032, torch.bfloat16, True), (297, 14336, torch.bfloat16, True),
                                            (890, 13824, torch.float16, False), (301, 16384, torch.bfloat16, True),
                                            (1185, 6152, torch.float16, True), (296, 8200, torch.bfloat16, False)])
def test_gelu_quantiser_bits(lib, M, K, dtype, bias):
    from instinctflash_b200.kernels import norm
    from oracle import oracle as O
    g = torch.Generator(device=DEV).manual_seed(M + K)
    x = (torch.randn(M, K, device=DEV, generator=g) * 30).to(dtype)
    row = torch.rand(M, device=DEV, generator=g) * 0.1
    col = torch.rand(K, device=DEV, generator=g) * 2
    b = torch.randn(K, device=DEV, generator=g) if bias else None
    outs = []
    for run in (lambda f: f(), lambda f: narrow(lib, f)):
        q, s = torch.full((M, K + 8), 1.0, device=DEV).to(E4M3), torch.empty(M, device=DEV)
        run(lambda: norm.row_quant(x, q[:, :K], s, row=row, col=col, bias=b, gelu=True))
        outs.append((q, s))
    torch.cuda.synchronize()
    assert torch.equal(u8(outs[0][0]), u8(outs[1][0])) and torch.equal(i32(outs[0][1]), i32(outs[1][1]))
    pick = torch.tensor([0, M // 2, M - 1], device=DEV)
    qo, so = O.row_quant(x[pick].cpu(), row=row[pick].cpu(), col=col.cpu(), bias=None if b is None else b.cpu(), gelu=True)
    assert_quant_close_to_oracle(outs[0][0][pick][:, :K], outs[0][1][pick], qo, so, f"{M}x{K}")


@pytest.mark.parametrize("M,D,delta,gate,affine", [(2960, 1032, True, True, "mod"), (593, 5120, True, True, "norm"),
                                                   (1777, 3072, True, False, "mod"), (300, 8192, True, True, "mod"),
                                                   (600, 5128, False, False, None), (1500, 2048, False, False, "mod")])
def test_residual_norm_rows(M, D, delta, gate, affine):
    from instinctflash_b200.kernels import norm
    from oracle import oracle as O
    g = torch.Generator(device=DEV).manual_seed(M + D)

    def randn(*shape, scale=1.0):
        return torch.randn(*shape, device=DEV, generator=g) * scale

    res = randn(M, D).to(torch.bfloat16)
    kw, per_row = {}, {}
    if delta:
        per_row = {"delta": randn(M, D, scale=100.0).to(torch.bfloat16), "delta_row": torch.rand(M, device=DEV, generator=g) * 0.02}
        kw = {"delta_col": randn(D), "bias": randn(D)}
    if gate:
        kw["gate"] = randn(D)
    if affine:
        names = ("mod_scale", "mod_shift") if affine == "mod" else ("weight", "beta")
        kw.update({names[0]: randn(D, scale=0.2), names[1]: randn(D, scale=0.2)})
    pick = torch.tensor([0, 1, M // 2, M - 2, M - 1], device=DEV)
    want = O.residual_norm_quant(res[pick].cpu(), layernorm=True, **{k: v[pick].cpu() for k, v in per_row.items()},
                                 **{k: v.cpu() for k, v in kw.items()})
    q, s = torch.full((M, D + 8), 1.0, device=DEV).to(E4M3), torch.full((M,), -1.0, device=DEV)
    norm.residual_norm_quant(res, layernorm=True, q=q[:, :D], q_scale=s, **per_row, **kw)
    torch.cuda.synchronize()
    assert (s > 0).all()
    assert torch.equal(res[pick].cpu(), want["res"])   # elementwise: no sum in it
    assert (q[:, D:].float() == 1.0).all()
    # the order of the two sums of D terms is free: D * 2^-24 each, well under 1e-5 of the scale here
    assert ((s[pick].cpu() - want["qs"]).abs() / want["qs"]).max().item() < 1e-5
    steps = code_steps(q[pick][:, :D], want["q"])
    assert steps.max().item() <= 1 and (steps != 0).float().mean().item() < 2e-3


# 1777 rows of 3072 take two turns of seven groups on 768 threads, the first 1480 of them two of five on 640: the same
# threads own a row, so its bits are the same
@pytest.mark.parametrize("gate", [False, True])
def test_residual_norm_rows_on_more_groups(gate):
    from instinctflash_b200.kernels import norm
    M, few, D = 1777, 1480, 3072
    g = torch.Generator(device=DEV).manual_seed(D)

    def randn(*shape, scale=1.0):
        return torch.randn(*shape, device=DEV, generator=g) * scale

    res, delta, row = randn(M, D).to(torch.bfloat16), randn(M, D, scale=100.0).to(torch.bfloat16), torch.rand(M, device=DEV, generator=g) * 0.02
    kw = {"delta_col": randn(D), "bias": randn(D), "mod_scale": randn(D, scale=0.2), "mod_shift": randn(D, scale=0.2)}
    if gate:
        kw["gate"] = randn(D)
    outs = []
    for rows in (M, few):
        r, q, s = res[:rows].clone(), torch.full((rows, D + 8), 1.0, device=DEV).to(E4M3), torch.full((rows,), -1.0, device=DEV)
        norm.residual_norm_quant(r, delta=delta[:rows], delta_row=row[:rows], layernorm=True, q=q[:, :D], q_scale=s, **kw)
        outs.append((r, u8(q), i32(s)))
    torch.cuda.synchronize()
    for all_rows, first_rows in zip(*outs):
        assert torch.equal(all_rows[:few], first_rows)
    assert (outs[0][2][few:] > 0).all() and (outs[0][1][:, D:] == 0x38).all()


# heads narrower than a thread's stride (its chunks lie at different pairs), one part only, no norm, pool slots
@pytest.mark.parametrize("B,T,H,HD,parts,norm,dtype", [(2, 700, 24, 128, 3, True, torch.float16), (1, 1801, 9, 120, 3, False, torch.bfloat16),
                                                       (1, 1900, 12, 128, 1, True, torch.bfloat16), (1, 593, 40, 128, 3, True, torch.float16)])
def test_wan_qkv_rows(lib, B, T, H, HD, parts, norm, dtype):
    from instinctflash_b200.kernels import rope, wan
    from oracle import oracle as O
    g = torch.Generator(device=DEV).manual_seed(T)
    D, R = H * HD, B * T
    raw = torch.randn(R, parts * D, device=DEV, generator=g).to(torch.bfloat16)
    row = torch.rand(R, device=DEV, generator=g)
    col, bias = torch.rand(parts * D, device=DEV, generator=g), torch.randn(parts * D, device=DEV, generator=g)
    w = {n: torch.rand(D, device=DEV, generator=g) + 0.5 if norm else None for n in ("q_norm", "k_norm")}
    pos = (torch.rand(T, 3, device=DEV, generator=g) * 60).floor()
    sec = (torch.arange(HD // 2, device=DEV) % 3).int()
    inv = rope.rope_inv_freq(HD, 10000.0, DEV)
    slots = torch.randperm(T, device=DEV, generator=g).int()
    q = torch.full((R, D + 8), 7.0, device=DEV, dtype=dtype)
    pools = [torch.empty(B, T, D, device=DEV, dtype=dtype) if parts > 1 + i else None for i in range(2)]
    wan.wan_qkv(raw, q[:, :D], heads=H, head_dim=HD, tokens=T, k_pool=pools[0], v_pool=pools[1], slots=slots, row=row, col=col,
                bias=bias, pos=pos, sections=sec, inv_freq=inv, **w)
    torch.cuda.synchronize()
    tok = torch.tensor([0, 1, T // 2, T - 1], device=DEV)
    for b in range(B):
        rows = b * T + tok
        want = O.wan_qkv(raw[rows].cpu(), heads=H, head_dim=HD, tokens=len(tok), parts=parts, row=row[rows].cpu(), col=col.cpu(),
                         bias=bias.cpu(), pos=pos[tok].cpu(), sections=sec.cpu(), inv_freq=inv.cpu(), out_dtype=dtype,
                         **{n: None if t is None else t.cpu() for n, t in w.items()})
        got = [q[rows][:, :D]] + [None if p is None else p[b][slots[tok].long()] for p in pools]
        ulp = 2.0 ** -10 if dtype == torch.float16 else 2.0 ** -7
        for i, (a, e) in enumerate(zip(got, want)):
            if a is None:
                continue
            a, e = a.cpu().float(), e.reshape(len(tok), D).float()
            if i == 2:
                assert torch.equal(a, e)   # V: no sum and no angle in it
            # one rounding of the output apart (the sum of squares is free in its order, sine and cosine are the
            # libraries'): relative to the pair's magnitude, since a rotation can cancel
            mag = e.reshape(-1, 2).norm(dim=1).repeat_interleave(2).reshape(e.shape)
            assert ((a - e).abs() <= ulp * mag + 1e-6).all(), (i, ((a - e).abs() / mag).max())
    assert (q[:, D:] == 7.0).all()


# one token; a CTA's tokens not whole, a unit round not whole; many tokens; wide heads; no norm (every bit then)
@pytest.mark.parametrize("T,HQ,HKV,HD,norm", [(1, 8, 1, 64, True), (3001, 5, 1, 64, True), (611, 12, 4, 128, False), (301, 10, 2, 256, True), (1501, 3, 2, 256, True),
                                              (2400, 16, 4, 64, False)])
def test_qkv_split_tokens_per_cta(lib, T, HQ, HKV, HD, norm):
    from instinctflash_b200.kernels import rope
    from oracle import oracle as O
    g = torch.Generator(device=DEV).manual_seed(T)
    W = (HQ + 2 * HKV) * HD
    raw = torch.randn(T, W, device=DEV, generator=g).to(torch.bfloat16)
    kw = dict(heads_q=HQ, heads_kv=HKV, head_dim=HD)
    per_row = dict(row=torch.rand(T, device=DEV, generator=g), pos=(torch.rand(T, 2, device=DEV, generator=g) * 900).floor())
    vec = dict(col=torch.rand(W, device=DEV, generator=g), bias=torch.randn(W, device=DEV, generator=g),
               inv_freq=rope.rope_inv_freq(HD, 10000.0, DEV), sections=(torch.arange(HD // 2, device=DEV) % 2).int())
    if norm:
        vec.update(q_norm=torch.rand(HD, device=DEV, generator=g) + 0.5, k_norm=torch.rand(HD, device=DEV, generator=g) + 0.5)
    q = torch.full((T, HQ, HD), 7.0, device=DEV, dtype=torch.float16)
    k, v = (torch.full((T + 9, HKV, HD), 7.0, device=DEV, dtype=torch.float16) for _ in range(2))
    rope.qkv_split(raw, q, k, v, kv_base=5, **kw, **per_row, **vec)
    torch.cuda.synchronize()
    pick = torch.tensor(sorted({0, T // 3, T - 1}), device=DEV)
    qo, ko, vo = O.qkv_split(raw[pick].cpu(), kv_rows=len(pick), **kw, **{n: t[pick].cpu() for n, t in per_row.items()},
                             **{n: t.cpu() for n, t in vec.items()})
    assert torch.equal(v[5 + pick].cpu(), vo)   # V: no sum and no angle in it
    for a, e in ((q[pick].cpu().float(), qo.float()), (k[5 + pick].cpu().float(), ko.float())):
        # a rounding of the output and one of sine or cosine, relative to the pair it rotates
        mag = torch.stack((e[..., :HD // 2], e[..., HD // 2:])).norm(dim=0).repeat(1, 1, 2)
        assert ((a - e).abs() <= 2.0 ** -10 * mag + 1e-6).all()
    assert (k[:5] == 7.0).all() and (v[5 + T:] == 7.0).all()

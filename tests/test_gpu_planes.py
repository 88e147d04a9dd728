"""Residual + norm + quantiser over the planes of a K-split GEMM: both kernel forms at the lines of the rule that
chooses between them, with every optional operand, against the oracle."""
import pytest
import torch

from util import code_steps, u8

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4M3 = torch.float8_e4m3fn


# one to eight quads of columns a thread, ragged last ones; rows in one wave, over it, in a second of either form;
# planes: one, a whole group, a group and one, all eight
@pytest.mark.parametrize("M,D,S", [(1, 8, 8), (50, 1024, 5), (300, 2056, 2), (444, 3072, 3), (445, 3072, 3), (593, 3064, 1), (816, 3072, 6),
                                   (816, 2056, 7), (5, 3080, 4), (301, 4096, 8), (33, 4104, 2), (33, 4104, 3), (600, 5120, 1),
                                   (7, 5128, 5), (129, 6152, 4), (300, 8192, 8)])
@pytest.mark.parametrize("kind", ["rms", "layer"])
def test_planes_of_every_width(M, D, S, kind):
    from instinctflash_b200.kernels import norm
    from oracle import oracle as O
    g = torch.Generator(device=DEV).manual_seed(M + D + S)

    def randn(*shape, scale=1.0):
        return torch.randn(*shape, device=DEV, generator=g) * scale

    layer = kind == "layer"
    res = randn(M, D).to(torch.bfloat16 if layer else torch.float32)
    planes, drow = randn(S, M, D, scale=40.0), torch.rand(M, device=DEV, generator=g) * 0.02
    kw = {"delta_col": randn(D)}
    if layer:
        kw.update(bias=randn(D), gate=randn(D), weight=randn(D), beta=randn(D, scale=0.2), mod_scale=randn(D, scale=0.2), mod_shift=randn(D, scale=0.2))
    total = planes[0].clone()
    for p in planes[1:]:
        total = total + p   # in plane order, then the accumulator's rounding point
    pick = torch.tensor(sorted({0, M // 2, M - 1}), device=DEV)
    want = O.residual_norm_quant(res[pick].cpu(), delta=total[pick].to(torch.bfloat16).cpu(), delta_row=drow[pick].cpu(), layernorm=layer,
                                 y_dtype=torch.float32, **{k: v.cpu() for k, v in kw.items()})
    q, s = torch.full((M, D + 8), 1.0, device=DEV).to(E4M3), torch.full((M,), -1.0, device=DEV)
    y = torch.full((M, D), float("nan"), device=DEV)
    norm.residual_norm_quant(res, delta=planes, delta_row=drow, layernorm=layer, q=q[:, :D], q_scale=s, y=y, **kw)
    torch.cuda.synchronize()
    assert (s > 0).all() and not torch.isnan(y).any() and (q[:, D:].float() == 1.0).all()
    assert torch.equal(res[pick].cpu(), want["res"])   # elementwise: no sum over the row in it
    # sums of D terms in another order: D * 2^-24 relative at the most, far less on average
    assert ((s[pick].cpu() - want["qs"]).abs() / want["qs"]).max().item() < 1e-5
    steps = code_steps(q[pick][:, :D], want["q"])
    assert steps.max().item() <= 1 and (steps != 0).float().mean().item() < 5e-3


@pytest.mark.parametrize("M,D,S", [(40, 3072, 8), (500, 3072, 4), (20, 5120, 8), (20, 8192, 2)])
def test_mirrors_hold_the_same_bits(M, D, S):
    from instinctflash_b200.kernels import norm
    g = torch.Generator(device=DEV).manual_seed(D)
    res = torch.randn(M, D, device=DEV, generator=g)
    planes = torch.randn(S, M, D, device=DEV, generator=g)
    q = [torch.zeros(M, D, device=DEV).to(E4M3) for _ in range(3)]
    s = [torch.zeros(M, device=DEV) for _ in range(3)]
    norm.residual_norm_quant_peers(res, delta=planes, q=q[0], q_scale=s[0], q_mirrors=q[1:], q_scale_mirrors=s[1:])
    torch.cuda.synchronize()
    assert (s[0] > 0).all()
    for k in (1, 2):
        assert torch.equal(u8(q[0]), u8(q[k])) and torch.equal(s[0], s[k])

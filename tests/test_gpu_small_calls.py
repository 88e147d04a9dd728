"""Small calls: the one-launch dynamic pack at the edges of its range against the two-kernel form, the
attention merge with more splits than one group of loads holds."""
import pytest
import torch

from util import assert_quant_close_to_oracle, i32, u8

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4M3 = torch.float8_e4m3fn


# one chunk; a CTA of the cluster empty; every count of register chunks and cluster size full, and one over
@pytest.mark.parametrize("n", [8, 8 * 1023, 65536, 65544, 131072, 131080, 262144, 262152, 524288, 524296])
@pytest.mark.parametrize("kind", ["normal", "zeros", "nan", "inf", "tiny"])
def test_one_launch_pack(n, kind):
    from instinctflash_b200 import _lib
    from instinctflash_b200.runtime.fp8_pack import dynamic_pack_bf16_e4m3
    g = torch.Generator(device=DEV).manual_seed(n)
    x = torch.randn(n, device=DEV, generator=g)
    x[::3] *= -0.0 if kind == "zeros" else 1e-3
    x = (x * (1e-38 if kind == "tiny" else 1.0)).to(torch.bfloat16)
    if kind in ("nan", "inf"):
        x[n - 1] = float(kind)
    if kind == "zeros":
        x = x * 0
    q, s = dynamic_pack_bf16_e4m3(x)
    q2, s2 = torch.empty(n, device=DEV, dtype=E4M3), torch.empty(1, device=DEV)
    assert _lib.lib().iflb200_dynamic_pack_bf16_e4m3_noalloc(x.data_ptr(), n, q2.data_ptr(), s2.data_ptr(),
                                                            torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert torch.equal(i32(s), i32(s2)) and torch.equal(u8(q), u8(q2))
    if kind == "normal":
        want = (x.float() / s).clamp(-448, 448).to(E4M3)   # the recipe's own division
        assert torch.equal(u8(q), u8(want))


@pytest.mark.parametrize("tokens,hq,hkv,hd,splits", [(3, 8, 1, 256, 9), (2, 16, 2, 64, 17), (1, 32, 8, 256, 8), (5, 4, 4, 20, 1), (70, 16, 4, 100, 3)])
def test_merge_of_more_splits_than_a_group(tokens, hq, hkv, hd, splits):
    from instinctflash_b200.kernels import attention
    from oracle import oracle as O
    g = torch.Generator(device=DEV).manual_seed(hd + splits)
    ws = attention.SplitWorkspace(1, tokens, hq, hkv, hd, splits, DEV)
    ws.po.normal_(generator=g)
    ws.pm.normal_(generator=g)
    ws.pl.uniform_(1.0, 50.0, generator=g)
    q8, s = torch.empty(tokens, hq * hd, device=DEV, dtype=E4M3), torch.empty(tokens, device=DEV)
    attention.attn_combine(ws, heads_q=hq, heads_kv=hkv, head_dim=hd, tokens=tokens, q8=q8, q8_scale=s)
    torch.cuda.synchronize()
    _, qo, so = O.attn_combine_quant(ws.po.cpu(), ws.pm.cpu(), ws.pl.cpu(), splits=splits, batch=1, tokens=tokens, heads_q=hq,
                                     heads_kv=hkv, head_dim=hd)
    # ex2.approx and div.full against the oracle's exp2f and division: the bounds of the recorded geometries
    assert_quant_close_to_oracle(q8, s, qo, so, f"{splits} splits", max_scale_ulp=16, max_code_frac=2e-2)

"""A projection module whose packed tensors a caller has replaced: by a parameter, by a plain attribute."""
import pytest
import torch

from instinctflash_b200.runtime import torch_fp8_linear as T


def as_parameter(m, name):
    t = getattr(m, name)
    delattr(m, name)
    setattr(m, name, torch.nn.Parameter(t, requires_grad=False))


def as_attribute(m, name):
    t = getattr(m, name)
    delattr(m, name)
    object.__setattr__(m, name, t)


REPLACED = [(how, name) for how in (as_parameter, as_attribute) for name in ("weight_fp8", "weight_scale", "bias")]


@pytest.mark.parametrize("how,name", REPLACED)
def test_replaced_buffer_is_found(monkeypatch, how, name):
    monkeypatch.setattr(T, "_target_device", lambda weight, *a: weight.device)
    m = T.SM100FP8Linear(torch.nn.Linear(32, 16, dtype=torch.bfloat16))
    seen = {}
    monkeypatch.setattr(T, "dynamic_pack_bf16_e4m3", lambda rows: (rows.to(torch.float8_e4m3fn), torch.ones(1)))
    monkeypatch.setattr(T, "fp8_linear", lambda a, s, w, out, **kw: seen.update(w=w, **kw))
    want = getattr(m, name)
    how(m, name)
    assert m(torch.zeros(3, 32, dtype=torch.bfloat16)).shape == (3, 16)
    used = {"weight_fp8": seen["w"].w, "weight_scale": seen["w"].scale, "bias": seen["bias"]}[name]
    assert used.data_ptr() == want.data_ptr()


@pytest.mark.gpu
@pytest.mark.parametrize("how,name", REPLACED)
def test_replaced_buffer_gives_the_same_bits(how, name):
    m = T.SM100FP8Linear(torch.nn.Linear(512, 48, device="cuda", dtype=torch.bfloat16))
    x = torch.randn(7, 512, device="cuda").to(torch.bfloat16)
    want = m(x)
    how(m, name)
    assert torch.equal(m(x), want)

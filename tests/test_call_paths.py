"""The library works without its native call path: a ``_calls.so`` that is missing, does not import or was built
against another torch costs host time per call, nothing else."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
BROKEN = {
    "missing": "sys.modules['instinctflash_b200._calls'] = None",
    "another torch": "import torch, instinctflash_b200._calls as c; c.torch_version = '1.0.0'",
}


def run(how, code):
    text = f"import sys, warnings; warnings.simplefilter('always'); {BROKEN[how]}\n{code}"
    env = {**os.environ, "PYTHONPATH": str(ROOT)}
    return subprocess.run([sys.executable, "-c", text], env=env, capture_output=True, text=True, timeout=600)


@pytest.mark.parametrize("how", sorted(BROKEN))
def test_library_loads_without_the_native_call_path(how):
    r = run(how, """
from instinctflash_b200 import _lib
assert _lib.lib().iflb200_abi_version() == _lib.ABI_VERSION
from instinctflash_b200.kernels import norm
""")
    assert r.returncode == 0, r.stderr
    assert "RuntimeWarning: the call path _calls.so is unavailable" in r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("how", sorted(BROKEN))
def test_operators_run_through_ctypes(how):
    r = run(how, """
import torch
from instinctflash_b200 import _lib
from instinctflash_b200.kernels import _common, fp8, norm
from instinctflash_b200.runtime.torch_fp8_linear import SM100FP8Linear
_lib.lib()
x = torch.randn(33, 256, device="cuda").to(torch.bfloat16)
q, s = torch.empty(33, 256, device="cuda", dtype=torch.float8_e4m3fn), torch.empty(33, device="cuda")
assert not _common.native.row_quant(x, q, s, None, None, None, False)
norm.row_quant(x, q, s)
assert ((q.float() * s[:, None] - x.float()).abs() <= x.float().abs() / 16 + s[:, None] * 2.0 ** -10).all()
m = torch.nn.Linear(256, 64, device="cuda", dtype=torch.bfloat16)
y = SM100FP8Linear(m)(x)
assert ((y - m(x)).float().norm() / m(x).float().norm()).item() < 0.1
""")
    assert r.returncode == 0, r.stderr

"""Shortened element functions against the long forms they replace, over all inputs: the kernels that use them are
tested against one another and against the oracle on samples only."""
import ctypes
import subprocess
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def checks(tmp_path_factory):
    from instinctflash_b200 import build
    so = tmp_path_factory.mktemp("exhaustive") / "exhaustive.so"
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-shared", "-I", str(ROOT / "instinctflash_b200" / "csrc"),
                    str(ROOT / "tests" / "exhaustive.cu"), "-o", str(so), "-Xcompiler", "-fvisibility=default"],
                   check=True, capture_output=True, text=True, timeout=600)
    return ctypes.CDLL(str(so))


# 0: GELU of two elements, all 2^32 floats; 1: codes of a per-tensor pack, every bf16 maximum (infinity and NaN
# among them) with every bf16 element up to it
@pytest.mark.parametrize("what,inputs", [(0, 1 << 32), (1, sum(2 * (best + 1) for best in range(0x8000)))])
def test_no_result_differs(checks, what, inputs):
    out = torch.zeros(3, device="cuda", dtype=torch.int64)
    torch.cuda.synchronize()
    assert checks.compare_all(what, ctypes.c_void_p(out.data_ptr())) == 0
    assert out[0].item() == 0, hex(out[1].item())
    assert out[2].item() == inputs

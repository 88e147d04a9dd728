"""Build ``libiflb200.so`` (sm_100a) in-tree with nvcc, and ``_calls.so`` (the call path from tensors
to it) with g++ against the installed torch.

Run as ``python -m instinctflash_b200.build`` or call :func:`build`.  nvcc cross-compiles
without a GPU.  Objects are cached by a hash of the sources and flags under ``csrc/_obj``.
"""
from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
INCLUDE = PKG.parent / "include"
LIBRARY = PKG / "libiflb200.so"
# (source, extra defines, object stem): row_ops.cu is compiled as three translation units in parallel
SOURCES = (("gemm_fp8_sm100.cu", (), "gemm_fp8_sm100"),
           ("stack_persistent.cu", (), "stack_persistent"),
           ("qkv_ops.cu", (), "qkv_ops"),
           ("attn_ops.cu", (), "attn_ops"),
           ("xgpu_ops.cu", (), "xgpu_ops"),
           ("row_stream.cu", (), "row_stream"),
           ("row_ops.cu", ("-DIFLB200_ROW_PART=0",), "row_ops_quant"),
           ("row_ops.cu", ("-DIFLB200_ROW_PART=1",), "row_ops_gated_pack"),
           ("row_ops.cu", ("-DIFLB200_ROW_PART=2",), "row_ops_resnorm"))
# the host call path: a CPython extension module over torch's headers
CALLS_SOURCE = "host_calls.cpp"
CALLS_MODULE = PKG / "_calls.so"
GXX_FLAGS = ("-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-w")
NVCC_FLAGS = (
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
)


def _nvcc() -> str:
    found = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(found).exists():
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build libiflb200.so")
    return found


def _digest(paths) -> str:
    h = hashlib.sha256()
    h.update(" ".join(NVCC_FLAGS).encode())
    for p in sorted(paths):
        h.update(p.name.encode())
        h.update(p.read_bytes())
    return h.hexdigest()[:16]


def _calls_job(force: bool, stamp: Path):
    """(command, tag) that builds ``_calls.so``, or (None, tag) when it is up to date."""
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths, library_paths

    src = CSRC / CALLS_SOURCE
    tag = _digest([src] + list(INCLUDE.glob("*.h"))) + f" torch {torch.__version__} " + " ".join(GXX_FLAGS)
    if not force and CALLS_MODULE.exists() and stamp.exists() and stamp.read_text() == tag:
        return None, tag
    cmd = ["g++", *GXX_FLAGS, str(src), "-o", str(CALLS_MODULE), "-I", sysconfig.get_paths()["include"]]
    for d in include_paths("cuda"):
        cmd += ["-isystem", d]
    for d in library_paths("cuda"):
        cmd += ["-L", d]
    cmd += ["-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]
    return cmd, tag


def build(force: bool = False, verbose: bool = False) -> Path:
    headers = list(CSRC.glob("*.cuh")) + list(INCLUDE.glob("*.h"))
    obj_dir = CSRC / "_obj"
    obj_dir.mkdir(exist_ok=True)
    nvcc = _nvcc()
    objects, jobs = [], []
    for name, defines, stem in SOURCES:
        src = CSRC / name
        tag = _digest([src] + headers)
        obj = obj_dir / f"{stem}.{tag}.o"
        objects.append(obj)
        if force or not obj.exists():
            for old in obj_dir.glob(f"{stem}.*.o"):
                old.unlink()
            cmd = [nvcc, *NVCC_FLAGS, *defines, "-I", str(INCLUDE), "-c", str(src), "-o", str(obj)]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"{Path(cmd[0]).name} failed: {' '.join(cmd)}\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)

    calls_stamp = obj_dir / "calls.stamp"
    calls_cmd, calls_tag = _calls_job(force, calls_stamp)
    compiled = bool(jobs)
    if calls_cmd:
        jobs.append(calls_cmd)
    if jobs:
        with ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 1)) as pool:
            list(pool.map(run, jobs))
    stamp = obj_dir / "link.stamp"
    want = " ".join(o.name for o in objects)
    if calls_cmd:
        calls_stamp.write_text(calls_tag)
    if compiled or not LIBRARY.exists() or not stamp.exists() or stamp.read_text() != want:
        run([nvcc, "-shared", "-Xcompiler", "-fPIC", "-o", str(LIBRARY), *map(str, objects)])
        stamp.write_text(want)
    return LIBRARY


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))

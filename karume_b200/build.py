"""Builds libkq.so in-tree with nvcc for sm_100a (cross-compiles without a GPU).

    python karume_b200/build.py [--verbose] [--force]

Every translation unit is compiled to an object file of its own (in parallel, and only when
it or a header changed), then linked.  The shared library lands next to this file so that it
travels with the source tree; nothing is installed into site-packages and nothing is
JIT-compiled at import time.
"""
from __future__ import annotations

import concurrent.futures
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
OUT = os.path.join(HERE, "libkq.so")
TORCH_SRC = os.path.join(CSRC, "kq_torch.cpp")
TORCH_OUT = os.path.join(HERE, "_kqtorch.so")  # the Python calls on torch tensors (a CPython extension module)

SOURCES = ["kq_api.cu", "kq_generic.cu", "kq_qgemv_i4.cu", "kq_qgemv_i4_xs.cu", "kq_qgemv_i4_tc.cu", "kq_qgemv_rows.cu", "kq_plan.cu", "kq_qgemm_i4.cu", "kq_qgemm_exact.cu", "kq_qgemv_i8.cu",
           "kq_comm.cu", "kq_idot.cu", "kq_fused_ops.cu", "kq_container.cu"]
HEADERS = ["kq_common.cuh", "kq_gemv_core.cuh", "kq_umma.cuh", "kq_gemm_stream.h", "kq_internal.h", "kq_per_device.h", "kq_exact_geometry.h", "kq_rows_line.h", os.path.join("..", "..", "include", "kq.h")]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
]


def _nvcc() -> str:
    found = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(found):
        raise RuntimeError("nvcc not found: libkq has no other build path")
    return found


def _newest_header() -> float:
    deps = [os.path.join(CSRC, h) for h in HEADERS] + [os.path.abspath(__file__)]
    return max(os.path.getmtime(d) for d in deps)


def _compile_one(args):
    src, obj, verbose, extra_flags = args
    cmd = [_nvcc(), *NVCC_FLAGS, *extra_flags, "-c", "-o", obj, src]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    if os.path.exists("/usr/bin/g++"):  # the distribution's g++ is the host compiler nvcc is validated with here
        cmd += ["-ccbin", "/usr/bin/g++"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    return src, proc.returncode, proc.stdout + proc.stderr, cmd


def build(force: bool = False, verbose: bool = False, extra_flags=(), out: str = OUT) -> str:
    os.makedirs(OBJ, exist_ok=True)
    headers = _newest_header()
    jobs, objects = [], []
    for s in SOURCES:
        src = os.path.join(CSRC, s)
        obj = os.path.join(OBJ, s.replace(".cu", ".o"))
        objects.append(obj)
        stale = force or extra_flags or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), headers)
        if stale:
            jobs.append((src, obj, verbose, tuple(extra_flags)))
    failed = []
    with concurrent.futures.ThreadPoolExecutor(max_workers=max(1, min(len(jobs), os.cpu_count() or 1))) as pool:
        for src, rc, log, cmd in pool.map(_compile_one, jobs):
            if verbose or rc != 0:
                sys.stderr.write(f"---- {os.path.basename(src)}\n{log}")
            if rc != 0:
                failed.append(" ".join(cmd))
    if failed:
        raise RuntimeError("nvcc failed:\n" + "\n".join(failed))
    if jobs or not os.path.exists(out) or out != OUT:
        cmd = [_nvcc(), "--shared", "-cudart", "shared", "-o", out, *objects]
        if os.path.exists("/usr/bin/g++"):
            cmd += ["-ccbin", "/usr/bin/g++"]
        proc = subprocess.run(cmd, capture_output=True, text=True)
        if proc.returncode != 0:
            sys.stderr.write(proc.stdout + proc.stderr)
            raise RuntimeError(f"link failed ({proc.returncode}): {' '.join(cmd)}")
    return out


def build_torch_calls(force: bool = False) -> str:
    """Compiles kq_torch.cpp against the torch of this interpreter (host code only)."""
    if not force and os.path.exists(TORCH_OUT) and os.path.getmtime(TORCH_OUT) >= max(os.path.getmtime(TORCH_SRC), os.path.getmtime(os.path.abspath(__file__))):
        return TORCH_OUT
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include"), sysconfig.get_paths()["include"]]
    lib = os.path.join(root, "lib")
    cmd = [shutil.which("g++") or "/usr/bin/g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for i in include:
        cmd += ["-isystem", i]
    cmd += ["-o", TORCH_OUT, TORCH_SRC, "-L" + lib, "-Wl,-rpath," + lib, "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        sys.stderr.write(proc.stdout + proc.stderr)
        raise RuntimeError(f"g++ failed ({proc.returncode}): {' '.join(cmd)}")
    return TORCH_OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
    print(build_torch_calls(force="--force" in sys.argv))

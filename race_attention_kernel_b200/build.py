"""Build the C-ABI shared library ``lib/librace_b200.so`` from ``csrc/*.cu`` with nvcc, and the torch host path
``_native.so`` (``csrc/torch_entry.cpp``, a CPython module that calls the library) with g++.

    python -m race_attention_kernel_b200.build [--force] [--verbose]

Targets sm_100a only (``-gencode arch=compute_100a,code=sm_100a``); nvcc cross-compiles, so
no GPU is needed to build.  Objects are rebuilt when a source or header is newer.
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIBDIR = os.path.join(HERE, "lib")
OBJDIR = os.path.join(HERE, "build")
LIB_PATH = os.path.join(LIBDIR, "librace_b200.so")
NATIVE_PATH = os.path.join(HERE, "_native.so")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-DRACE_B200", "-Xcompiler", "-fPIC", "-Xptxas", "-v",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _newest_header() -> float:
    t = 0.0
    for d in (CSRC, INCLUDE):
        for f in os.listdir(d):
            if f.endswith((".h", ".cuh")):
                t = max(t, os.path.getmtime(os.path.join(d, f)))
    return t


def build_native(force: bool = False) -> str:
    import sysconfig

    src = os.path.join(CSRC, "torch_entry.cpp")
    header = os.path.join(INCLUDE, "race_b200.h")
    if (not force and os.path.exists(NATIVE_PATH)
            and os.path.getmtime(NATIVE_PATH) >= max(os.path.getmtime(src), os.path.getmtime(header))):
        return NATIVE_PATH
    import torch

    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           "-I", INCLUDE, "-I", os.path.join(root, "include"), "-I", os.path.join(root, "include/torch/csrc/api/include"),
           "-I", sysconfig.get_paths()["include"], "-I", os.path.join(cuda, "include"), src, "-o", NATIVE_PATH,
           "-L", LIBDIR, "-lrace_b200", "-Wl,-rpath,$ORIGIN/lib", "-L", os.path.join(root, "lib"),
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", "-L", os.path.join(cuda, "lib64"), "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("g++ failed for torch_entry.cpp")
    return NATIVE_PATH


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(LIBDIR, exist_ok=True)
    os.makedirs(OBJDIR, exist_ok=True)
    sources = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
    hdr_t = _newest_header()
    nvcc = _nvcc()
    jobs = []
    objs = []
    for src in sources:
        sp = os.path.join(CSRC, src)
        op = os.path.join(OBJDIR, src[:-3] + ".o")
        objs.append(op)
        if force or not os.path.exists(op) or os.path.getmtime(op) < max(os.path.getmtime(sp), hdr_t):
            jobs.append((src, [nvcc, *NVCC_FLAGS, "-I", INCLUDE, "-c", sp, "-o", op]))

    def run(job):
        name, cmd = job
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode != 0:
            sys.stderr.write(f"--- {name}\n{r.stdout}{r.stderr}\n")
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {name}")
        return r.stderr

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        logs = list(ex.map(run, jobs))
    if jobs:
        with open(os.path.join(OBJDIR, "ptxas.log"), "a") as fh:
            for (name, _), log in zip(jobs, logs):
                fh.write(f"--- {name}\n{log}\n")
    if jobs or not os.path.exists(LIB_PATH):
        cmd = [nvcc, "-shared", "-o", LIB_PATH, *objs, "-gencode", "arch=compute_100a,code=sm_100a",
               "-lcuda"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    build_native(force)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))

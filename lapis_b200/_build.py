"""Builds ``liblapis_b200.so`` (nvcc, sm_100a) and the ``_calls`` extension module in-tree.

    python -m lapis_b200._build [--verbose]

Cross-compiles without a GPU.  The shared library sits beside this file so that
it travels with the source tree; nothing is installed into site-packages.
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "liblapis_b200.so")
CALLS = os.path.join(HERE, "_calls" + sysconfig.get_config_var("EXT_SUFFIX"))
SOURCES = ["abi.cu", "stage.cu", "spmv.cu", "spmm.cu", "pcg.cu", "pcg_small.cu", "pcg_grid.cu", "gemm.cu", "gemm_tcgen05.cu", "gemm_split.cu", "mmio.cu", "formats.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--fmad=false",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isfile(cand) or cand == "nvcc"):
            return cand
    raise RuntimeError("nvcc not found")


def needs_build() -> bool:
    if not os.path.isfile(LIB) or not os.path.isfile(CALLS):
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(CALLS))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    deps.append(os.path.join(os.path.dirname(HERE), "include", "lapis_b200.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def build(verbose: bool = False, force: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    objs = []
    env = dict(os.environ)
    env.pop("CC", None)
    env.pop("CXX", None)
    procs = [("torch_calls.cpp", _start_calls(env))]
    for src in SOURCES:
        obj = os.path.join(CSRC, src.replace(".cu", ".o"))
        cmd = [_nvcc(), *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
            print(" ".join(cmd), flush=True)
        procs.append((src, subprocess.Popen(cmd, env=env, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            print(out)
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    link = [_nvcc(), "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-lcuda"]
    subprocess.run(link, check=True, env=env)
    _link_calls(env)
    return LIB


def _start_calls(env):
    """Compiles the extension module (host compiler, torch's headers)."""
    from torch.utils import cpp_extension
    inc = [f"-I{p}" for p in cpp_extension.include_paths("cuda")] + [f"-I{sysconfig.get_paths()['include']}"]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", *inc, "-c", os.path.join(CSRC, "torch_calls.cpp"), "-o",
           os.path.join(CSRC, "torch_calls.o")]
    return subprocess.Popen(cmd, env=env, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def _link_calls(env):
    import torch
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = ["g++", "-shared", "-o", CALLS, os.path.join(CSRC, "torch_calls.o"), f"-L{HERE}", f"-l:{os.path.basename(LIB)}", f"-L{libs}",
           "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"]
    subprocess.run(cmd, check=True, env=env)


if __name__ == "__main__":
    print(build(verbose="--verbose" in sys.argv, force=True))

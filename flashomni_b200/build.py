"""Builds libflashomni_b200.so in-tree with nvcc for sm_100a.

    python -m flashomni_b200.build [--force] [--verbose]

and, with the host compiler, flashomni_b200/lib/_fo_host.so (csrc/host.cpp), the Python extension that issues the usual calls.
Each .cu under csrc/ is compiled to an object file (in parallel) and the objects are linked into
flashomni_b200/lib/libflashomni_b200.so. Objects are rebuilt when their source or any header is
newer. No GPU is needed to build.
"""

from __future__ import annotations

import argparse
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

from . import _native

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIBDIR = os.path.join(HERE, "lib")
OBJDIR = os.path.join(HERE, "lib", "obj")
LIB = os.path.join(LIBDIR, "libflashomni_b200.so")
SOURCES = ["api.cu", "masks.cu", "gemm.cu", "attention.cu", "attention_streams.cu", "static_scratch.cu", "exchange.cu", "select.cu", "gemm_tall.cu"]

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
          "--expt-relaxed-constexpr"]


HOST_SRC = os.path.join(CSRC, "host.cpp")
HOST_LIB = os.path.join(LIBDIR, "_fo_host.so")
HOST_STAMP = os.path.join(OBJDIR, "_fo_host.stamp")   # the command it was built with


def _host_cmd():
    import sysconfig
    import torch
    t = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(NVCC))
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
            f'-DFO_HOST_ABI="{_native.host_abi()}"',
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", f"-I{t}/include",
            f"-I{t}/include/torch/csrc/api/include", f"-I{sysconfig.get_paths()['include']}", f"-I{cuda}/include", HOST_SRC,
            "-o", HOST_LIB, f"-L{t}/lib", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda", f"-L{cuda}/lib64",
            "-lcudart"]


def _host_stamp() -> str:
    return " ".join(_host_cmd()) + "\n"


def _host_stale() -> bool:
    """The extension depends on the C++ interfaces of torch and Python, which change without any source here getting newer."""
    if _stale(HOST_LIB, [HOST_SRC, os.path.join(HERE, "..", "include", "flashomni_b200.h")]):
        return True
    try:
        with open(HOST_STAMP) as f:
            return f.read() != _host_stamp()
    except OSError:
        return True


def _headers():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    hs.append(os.path.join(HERE, "..", "include", "flashomni_b200.h"))
    return hs


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJDIR, exist_ok=True)
    headers = _headers()
    sources = [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]
    jobs = []
    for src in sources:
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJDIR, src.replace(".cu", ".o"))
        if force or _stale(o, [s] + headers):
            cmd = [NVCC, *ARCH_FLAGS, *COMMON, "-c", s, "-o", o]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)
    cuda_jobs = len(jobs)
    host = force or _host_stale()
    if host:
        if os.path.exists(HOST_STAMP):
            os.remove(HOST_STAMP)
        jobs.append(_host_cmd())

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    if jobs:
        with ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4)) as ex:
            for cmd, r in ex.map(run, jobs):
                if verbose or r.returncode != 0:
                    sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
                if r.returncode != 0:
                    raise RuntimeError(f"{os.path.basename(cmd[0])} failed: " + " ".join(cmd[-3:]))
    if host:
        with open(HOST_STAMP, "w") as f:
            f.write(_host_stamp())
    objs = [os.path.join(OBJDIR, s.replace(".cu", ".o")) for s in sources]
    if force or cuda_jobs or _stale(LIB, objs):
        cmd = [NVCC, *ARCH_FLAGS, "-shared", "-cudart", "shared", "-o", LIB, *objs,
               "-Xlinker", "-rpath", "-Xlinker", "/usr/local/cuda/lib64"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
            raise RuntimeError("link failed")
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))

"""Builds libshrewq.so (the C-ABI library) in-tree with nvcc for sm_100a, and _host.so (the per-call host path of the
Python mirror, a CPython extension) with the host compiler.

    python -m shrew_b200.build [--force] [--verbose] [--trace]

nvcc cross-compiles without a GPU.  The shared objects land beside this file so that they
travel with the source tree; nothing is written outside the package directory.
"""
from __future__ import annotations

import importlib.metadata
import os
import re
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libshrewq.so")
HOST_EXT = os.path.join(HERE, "_host.so")
SOURCES = ["api.cu", "quantize.cu", "quantize_batch.cu", "quantize_modes.cu", "gemv.cu", "gemv_mma.cu", "gemm_simt.cu", "gemm_tcgen05.cu", "gemm_tcgen05_g1.cu", "gemm_tcgen05_g2.cu", "gemm_tcgen05_g3.cu", "gemm_tcgen05_2cta.cu", "gemm_tcgen05_f32.cu", "exchange.cu"]
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
         "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden"]


def _includes(path: str, seen: set | None = None) -> list[str]:
    """The file and every header it includes by a quoted name, transitively: what its object depends on."""
    seen = set() if seen is None else seen
    if path not in seen and os.path.exists(path):
        seen.add(path)
        with open(path) as f:
            for name in re.findall(r'^\s*#\s*include\s+"([^"]+)"', f.read(), flags=re.M):
                _includes(os.path.normpath(os.path.join(os.path.dirname(path), name)), seen)
    return sorted(seen)


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_library(force: bool = False, verbose: bool = False, trace: bool = False) -> str:
    """trace=True builds libshrewq_trace.so: the same library with -DSHREWQ_TRACE, whose
    tcgen05 kernel stamps clock64() per pipeline role and stage."""
    if trace:
        return _build(os.path.join(CSRC, "build_trace"), os.path.join(HERE, "libshrewq_trace.so"),
                      FLAGS + ["-DSHREWQ_TRACE"], force, verbose)
    lib = _build(os.path.join(CSRC, "build"), LIB, FLAGS, force, verbose)
    build_host_extension(force, verbose)
    return lib


def _build(objdir: str, lib: str, flags: list[str], force: bool, verbose: bool) -> str:
    os.makedirs(objdir, exist_ok=True)
    jobs = []
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        o = os.path.join(objdir, src.replace(".cu", ".o"))
        if force or _stale(o, _includes(s)):
            cmd = [NVCC, *flags, "-c", s, "-o", o]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode != 0:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed: " + " ".join(cmd))

    with ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 1) or 1) as ex:
        list(ex.map(run, jobs))
    objs = [os.path.join(objdir, s.replace(".cu", ".o")) for s in SOURCES]
    if force or jobs or _stale(lib, objs):
        run([NVCC, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", lib, *objs, "-cudart", "static"])
    return lib


def build_host_extension(force: bool = False, verbose: bool = False) -> str:
    """_host.so: csrc/host_path.cpp against the headers and libraries of the installed torch."""
    src, stamp = os.path.join(CSRC, "host_path.cpp"), os.path.join(CSRC, "build", "host_extension.txt")
    against = f"torch {importlib.metadata.version('torch')}, python {sys.version.split()[0]}"   # what a built one matches
    built = open(stamp).read() if os.path.exists(stamp) else ""
    if not force and built == against and not _stale(HOST_EXT, _includes(src)):
        return HOST_EXT
    compile_host_extension(HOST_EXT, verbose=verbose)
    os.makedirs(os.path.dirname(stamp), exist_ok=True)
    with open(stamp, "w") as f:
        f.write(against)
    return HOST_EXT


def compile_host_extension(out: str, flags: list[str] | None = None, verbose: bool = False) -> None:
    """host_path.cpp with `flags` into the shared object `out` (the CPU tests build one of their own)."""
    src = os.path.join(CSRC, "host_path.cpp")
    import torch
    root = os.path.dirname(torch.__file__)
    cuda_inc = os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[a for d in (os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
                         sysconfig.get_paths()["include"], cuda_inc) for a in ("-isystem", d)],
           *(flags or []), src, "-o", out, "-L" + os.path.join(root, "lib"), "-Wl,-rpath," + os.path.join(root, "lib"),
           "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode != 0:
        sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError("host extension failed to build: " + " ".join(cmd))


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="--verbose" in sys.argv, trace="--trace" in sys.argv))

"""Build libevoattn.so (nvcc, sm_100a; cross-compiles without a GPU) and the native autograd boundary
_evohost.so (the host compiler, against the installed torch) in-tree.

    python -m evoformer_triton_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(PKG, "build")
LIB = os.path.join(PKG, "libevoattn.so")
HOST = os.path.join(PKG, "_evohost.so")
SOURCES = ["api.cu", "generic_kernels.cu", "tmap.cu", "fwd_sm100.cu", "bwd_sm100.cu", "peer_reduce.cu", "extras.cu"]
NVCC_FLAGS = [
    "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xptxas", "-v", "--expt-relaxed-constexpr",
    "-I", os.path.join(ROOT, "include"), "-I", CSRC,
] + os.environ.get("EVOATTN_NVCC_FLAGS", "").split()


def _nvcc() -> str:
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if c and (os.path.isabs(c) and os.path.exists(c) or not os.path.isabs(c)):
            return c
    return "nvcc"


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _host_flags():
    """Compiler and linker flags of the torch extension (torch's libraries are found at run time among
    those that ``import torch`` has loaded)."""
    import sysconfig
    import torch
    base = os.path.dirname(torch.__file__)
    cuda = os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")
    inc = [os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"), cuda, sysconfig.get_paths()["include"], os.path.join(ROOT, "include")]
    cxx = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_evohost"]
    cxx += [f for d in inc for f in ("-isystem", d)]
    return cxx, ["-L", os.path.join(base, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10"]


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(ROOT, "include", "evoattn.h"))
    jobs = []
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJ, src.replace(".cu", ".o"))
        if force or _stale(o, [s] + headers):
            jobs.append((s, o))

    host_src = os.path.join(CSRC, "host.cpp")
    host_obj = os.path.join(OBJ, "host.o")
    host_job = force or _stale(host_obj, [host_src, headers[-1]])
    cxx, ld = _host_flags()
    if host_job:
        jobs.append((host_src, host_obj))

    def compile_one(job):
        s, o = job
        cmd = ["g++", *cxx, "-c", s, "-o", o] if s == host_src else [_nvcc(), *NVCC_FLAGS, "-c", s, "-o", o]
        r = subprocess.run(cmd, capture_output=True, text=True)
        with open(o + ".log", "w") as f:
            f.write(r.stdout + r.stderr)
        return s, r

    with cf.ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for s, r in ex.map(compile_one, jobs):
            if verbose:
                sys.stderr.write(r.stderr)
            if r.returncode != 0:
                raise RuntimeError(f"compiling {s} failed:\n{r.stderr[-8000:]}")
    objs = [os.path.join(OBJ, s.replace(".cu", ".o")) for s in SOURCES]
    if force or any(s != host_src for s, _ in jobs) or _stale(LIB, objs):
        r = subprocess.run([_nvcc(), "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"],
                           capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n" + r.stderr[-4000:])
    if host_job or _stale(HOST, [host_obj]):
        r = subprocess.run(["g++", "-shared", "-o", HOST, host_obj, "-L", PKG, "-l:libevoattn.so", "-Wl,-rpath,$ORIGIN", *ld], capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n" + r.stderr[-4000:])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))

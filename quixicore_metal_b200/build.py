"""Builds the in-tree CUDA shared library for sm_100a with nvcc (no JIT cache).

    python -m quixicore_metal_b200.build            # incremental
    python -m quixicore_metal_b200.build --force    # rebuild everything

Objects go to quixicore_metal_b200/lib/obj, the result is quixicore_metal_b200/lib/libquixicore_cuda.so
(no torch headers) and, where torch is importable, lib/_qx_native.so: the C++ side of the Python binding.
"""
from __future__ import annotations

import concurrent.futures as cf
import glob
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIBDIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIBDIR, "libquixicore_cuda.so")
BINDING = os.path.join(LIBDIR, "_qx_native.so")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the CUDA toolkit is required to build quixicore_metal_b200")


def _newest_header() -> float:
    hs = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + \
        glob.glob(os.path.join(INCLUDE, "*.h"))
    return max(os.path.getmtime(h) for h in hs)


def build(force: bool = False, verbose: bool = False) -> str:
    nvcc = _nvcc()
    objdir = os.path.join(LIBDIR, "obj")
    os.makedirs(objdir, exist_ok=True)
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    hdr_time = _newest_header()
    jobs = []
    objs = []
    for src in sources:
        obj = os.path.join(objdir, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        stale = force or not os.path.exists(obj) or \
            os.path.getmtime(obj) < max(os.path.getmtime(src), hdr_time)
        if stale:
            jobs.append([nvcc, *NVCC_FLAGS, "-Xptxas", "-v", "-c", src, "-o", obj])

    def run(cmd):
        p = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, p.returncode, p.stdout + p.stderr

    if jobs:
        with cf.ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            for cmd, rc, out in ex.map(run, jobs):
                name = os.path.basename(cmd[-3])
                with open(os.path.join(objdir, name + ".ptxas.log"), "w") as f:
                    f.write(out)
                if rc != 0:
                    raise RuntimeError(f"nvcc failed for {name}:\n{out[-4000:]}")
                if verbose:
                    print(out)
    if jobs or not os.path.exists(LIB):
        cmd = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
        p = subprocess.run(cmd, capture_output=True, text=True)
        if p.returncode != 0:
            raise RuntimeError("link failed:\n" + p.stdout + p.stderr)
    build_binding(force)
    return LIB


def build_binding(force: bool = False) -> None:
    """lib/_qx_native.so from csrc/qx_binding.cpp.  A host without torch has no use for it."""
    src = os.path.join(CSRC, "qx_binding.cpp")
    header = os.path.join(INCLUDE, "quixicore_cuda.h")
    if not force and os.path.exists(BINDING) and os.path.getmtime(BINDING) >= max(os.path.getmtime(src), os.path.getmtime(header)):
        return
    try:
        import torch
    except ImportError:
        return
    import sysconfig
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_path("include"), os.path.join(cuda, "include")]
    cmd = [os.environ.get("CXX") or shutil.which("g++") or "c++", "-O2", "-std=c++17", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-o", BINDING, src,
           *[f"-I{d}" for d in inc], f"-L{os.path.join(root, 'lib')}", f"-L{LIBDIR}", "-lquixicore_cuda", "-ltorch",
           "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-ltorch_python", "-Wl,-rpath,$ORIGIN"]
    p = subprocess.run(cmd, capture_output=True, text=True)
    if p.returncode != 0:
        raise RuntimeError("binding build failed:\n" + (p.stdout + p.stderr)[-4000:])


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))

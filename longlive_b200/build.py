"""In-tree build of ``libllnvfp4.so`` (the C-ABI library) with nvcc for sm_100a, and of ``_native.so``
(its Python binding) with g++ against the installed PyTorch.

``python -m longlive_b200.build`` compiles every ``csrc/*.cu`` into one object each (in
parallel) and links them into ``longlive_b200/libllnvfp4.so``, then ``csrc/binding.cpp`` into
``longlive_b200/_native.so``.  Objects are rebuilt only when a source or header is newer, the binding
also when PyTorch, Python or its compile command is another.  nvcc cross-compiles without a GPU.
"""
from __future__ import annotations

import concurrent.futures as cf
import glob
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(PKG, "build")
LIB = os.path.join(PKG, "libllnvfp4.so")
NATIVE = os.path.join(PKG, "_native.so")
NATIVE_STAMP = os.path.join(OBJ, "_native.stamp")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: set NVCC or put it on PATH")


def _newest(paths) -> float:
    return max(os.path.getmtime(p) for p in paths)


def _build_binding(verbose: bool, force: bool) -> None:
    import sysconfig
    import torch
    from torch.utils.cpp_extension import include_paths, library_paths
    src = os.path.join(CSRC, "binding.cpp")
    cuda_home = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    inc = [*include_paths(), os.path.join(cuda_home, "include"), sysconfig.get_paths()["include"]]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_native",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DLLNV_TORCH_VERSION="{torch.__version__}"',
           *(f"-isystem{p}" for p in inc), src, "-o", NATIVE,
           f"-L{PKG}", "-lllnvfp4", "-Wl,-rpath,$ORIGIN", *(f"-L{p}" for p in library_paths()), "-lc10", "-lc10_cuda", "-ltorch_cpu",
           "-ltorch", "-ltorch_python"]
    # what the binary was built for and how: it is tied to one PyTorch and one Python, which no source time shows
    stamp = "\n".join([torch.__version__, sysconfig.get_config_var("SOABI") or "", *(a.replace(PKG, "<pkg>") for a in cmd)])
    newest = _newest([src, os.path.join(PKG, "..", "include", "llnvfp4.h")])
    if not force and os.path.exists(NATIVE) and os.path.getmtime(NATIVE) >= newest and os.path.exists(NATIVE_STAMP):
        with open(NATIVE_STAMP) as f:
            if f.read() == stamp:
                return
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode != 0:
        sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError("build of _native.so failed")
    os.makedirs(OBJ, exist_ok=True)
    with open(NATIVE_STAMP, "w") as f:
        f.write(stamp)


def build(verbose: bool = False, force: bool = False) -> str:
    nvcc = _nvcc()
    os.makedirs(OBJ, exist_ok=True)
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(PKG, "..", "include", "*.h"))
    hdr_time = _newest(headers) if headers else 0.0
    jobs = []
    objs = []
    for src in sources:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), hdr_time):
            cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    with cf.ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for cmd, r in ex.map(run, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
            if r.returncode != 0:
                raise RuntimeError(f"nvcc failed for {cmd[-3]}")
    if jobs or not os.path.exists(LIB) or os.path.getmtime(LIB) < _newest(objs):
        cmd = [nvcc, "-shared", "-o", LIB, *objs, "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link of libllnvfp4.so failed")
    _build_binding(verbose, force)
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))

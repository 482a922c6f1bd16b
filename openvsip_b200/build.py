"""Build the fcb200 CUDA library in-tree (sm_100a) with nvcc.

The library is openvsip_b200/libfcb200.so; translation units are compiled in
parallel into openvsip_b200/_build/.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libfcb200.so")

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
         f"-I{os.path.join(ROOT, 'include')}", f"-I{CSRC}"]

SOURCES = ["fcb_rows_conv.cu", "fcb_rows_coefs.cu", "fcb_rows_fwd.cu", "fcb_rows_inv.cu", "fcb_rows_r2c.cu",
           "fcb_rows_c2r.cu", "fcb_rows_cross.cu", "fcb_batch.cu", "fcb_mixed_conv.cu", "fcb_mixed_rows.cu",
           "fcb_mixed_cols.cu", "fcb_mixed.cu", "fcb200.cu",
           "fcb_api.cu", "fcb_bluestein.cu", "fcb_real.cu", "fcb_hostcopy.cu"]


def nvcc() -> str:
    path = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(path):
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build libfcb200.so")
    return path


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _headers() -> list[str]:
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs.append(os.path.join(ROOT, "include", "fcb200.h"))
    return hs


def build(verbose: bool = False, force: bool = False) -> str:
    os.makedirs(BUILD, exist_ok=True)
    headers = _headers()
    srcs = [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]
    jobs = []
    objs = []
    for s in srcs:
        src = os.path.join(CSRC, s)
        obj = os.path.join(BUILD, s.replace(".cu", ".o"))
        objs.append(obj)
        if force or _stale(obj, [src] + headers):
            cmd = [nvcc(), *ARCH, *FLAGS, "-c", src, "-o", obj]
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed: {' '.join(cmd)}\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stdout.write(r.stdout + r.stderr)
        return cmd

    with cf.ThreadPoolExecutor(max_workers=max(1, min(len(jobs), os.cpu_count() or 1))) as ex:
        list(ex.map(run, jobs))
    if force or jobs or _stale(LIB, objs):
        cmd = [nvcc(), *ARCH, "-shared", "-o", LIB, *objs, "-lcudart", "-lpthread"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed: {' '.join(cmd)}\n{r.stdout}\n{r.stderr}")
    return LIB


def build_torch(force: bool = False) -> str:
    """The native host path for CUDA tensors (csrc/fcb_torch.cpp), a Python
    extension module against the installed torch: built again when that or the
    Python changes (_fcb_torch.tag says what it was built for)."""
    import sysconfig

    import torch

    from ._lib import torch_tag
    src = os.path.join(CSRC, "fcb_torch.cpp")
    out, tag = os.path.join(HERE, "_fcb_torch.so"), os.path.join(HERE, "_fcb_torch.tag")
    built_for = open(tag).read() if os.path.exists(tag) else ""
    if not force and not _stale(out, [src]) and built_for == torch_tag():
        return out
    tdir = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc())))
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DFCB_BUILT_FOR="{torch_tag()}"',
           f"-I{sysconfig.get_paths()['include']}", f"-I{tdir}/include", f"-I{tdir}/include/torch/csrc/api/include",
           f"-I{cuda}/include", src, "-o", out, f"-L{tdir}/lib", "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed: {' '.join(cmd)}\n{r.stdout}\n{r.stderr}")
    with open(tag, "w") as f:
        f.write(torch_tag())
    return out


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))
    print(build_torch(force="-f" in sys.argv))

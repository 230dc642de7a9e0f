"""Builds libjvpfa.so (the C-ABI CUDA library, nvcc for sm_100a) and _host.so (the native host path, g++) in-tree.

Usage: ``python -m jvp_flash_attention_b200.build [--force] [--verbose]``. Each ``csrc/*.cu`` is
compiled to an object (in parallel) and linked into ``jvp_flash_attention_b200/libjvpfa.so``.
Objects are rebuilt only when a source or header is newer than them.
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = PKG / "csrc" / "build"
LIB = PKG / "libjvpfa.so"
HOST_SRC = CSRC / "host_torch.cpp"      # the native host path: plain C++ against torch, no CUDA code
HOST_LIB = PKG / "_host.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "-Xptxas", "-v",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found; set NVCC")


def _newest_header_mtime() -> float:
    hdrs = list(CSRC.glob("*.h")) + list(CSRC.glob("*.cuh")) + list((PKG.parent / "include").glob("*.h"))
    return max(h.stat().st_mtime for h in hdrs)


def _build_host() -> None:
    import sysconfig
    import torch
    from torch.utils.cpp_extension import CUDA_HOME, include_paths, library_paths
    inc = [f"-I{p}" for p in (*include_paths(), sysconfig.get_paths()["include"], f"{CUDA_HOME or '/usr/local/cuda'}/include")]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *inc, str(HOST_SRC), "-o", str(HOST_LIB),
           *(f"-L{p}" for p in library_paths()), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError(f"g++ failed on {HOST_SRC.name}")


def build(force: bool = False, verbose: bool = False) -> Path:
    nvcc = _nvcc()
    OBJ.mkdir(parents=True, exist_ok=True)
    srcs = sorted(CSRC.glob("*.cu"), key=lambda f: ("bwd" not in f.name, f.name))      # the long compilations first
    hdr_m = _newest_header_mtime()
    jobs = []
    for src in srcs:
        obj = OBJ / (src.stem + ".o")
        if force or not obj.exists() or obj.stat().st_mtime < max(src.stat().st_mtime, hdr_m):
            jobs.append((src, obj))

    def compile_one(job):
        src, obj = job
        cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        return src, r

    host_stale = force or not HOST_LIB.exists() or HOST_LIB.stat().st_mtime < max(HOST_SRC.stat().st_mtime, hdr_m)
    with ThreadPoolExecutor(max_workers=min(8, len(jobs) + 1)) as ex:
        host_job = ex.submit(_build_host) if host_stale else None
        for src, r in ex.map(compile_one, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(f"--- {src.name}\n{r.stdout}{r.stderr}\n")
            (OBJ / (src.stem + ".ptxas.txt")).write_text(r.stderr)
            if r.returncode != 0:
                raise RuntimeError(f"nvcc failed on {src.name}")
        if host_job is not None:
            host_job.result()
    objs = [str(OBJ / (s.stem + ".o")) for s in srcs]
    if jobs or not LIB.exists() or force:
        cmd = [nvcc, "-shared", "-o", str(LIB), *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))

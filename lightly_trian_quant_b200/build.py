"""Builds the C-ABI shared library (libkf_b200.so) in-tree with nvcc for sm_100a, and the native operator module on top of it
(_kf_host, a CPython extension that uses torch's C++ headers) with the host compiler.

    python -m lightly_trian_quant_b200.build [--force] [--verbose]

nvcc cross-compiles without a GPU.  Objects are cached under csrc/build/ keyed by a hash of each source and the
shared headers, so an unchanged file is not recompiled.  What ptxas says about registers and spills stays beside each object (.ptxas).
"""
from __future__ import annotations

import hashlib
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libkf_b200.so"
HOST_SRC = CSRC / "host" / "kf_host.cpp"
HOST_LIB = PKG / ("_kf_host" + sysconfig.get_config_var("EXT_SUFFIX"))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo", "--expt-relaxed-constexpr",
         "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "-Xptxas", "-v", "-DKF_BUILD"]


def sources():
    return sorted(CSRC.glob("*.cu"))


def _headers_hash() -> str:
    h = hashlib.sha256()
    for p in sorted(CSRC.glob("*.cuh")) + sorted((PKG.parent / "include").glob("*.h")):
        h.update(p.read_bytes())
    h.update(" ".join(FLAGS).encode())
    return h.hexdigest()


def build(force: bool = False, verbose: bool = False) -> Path:
    bdir = CSRC / "build"
    bdir.mkdir(exist_ok=True)
    hh = _headers_hash()
    jobs = []
    objs = []
    for src in sources():
        tag = hashlib.sha256(src.read_bytes() + hh.encode()).hexdigest()[:16]
        obj = bdir / f"{src.stem}.{tag}.o"
        objs.append(obj)
        if force or not (obj.exists() and obj.with_suffix(".ptxas").exists()):
            for old in [*bdir.glob(f"{src.stem}.*.o"), *bdir.glob(f"{src.stem}.*.ptxas")]:
                old.unlink()
            jobs.append((src, obj))

    def compile_one(job):
        src, obj = job
        cmd = [NVCC, *FLAGS, "-c", str(src), "-o", str(obj)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stdout}\n{r.stderr}")
        obj.with_suffix(".ptxas").write_text(r.stderr)
        if verbose:
            print(r.stderr)
        return obj

    if jobs:
        with ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            list(ex.map(compile_one, jobs))
    if jobs or force or not LIB.exists():
        cmd = [NVCC, "-shared", "-o", str(LIB), *map(str, objs), "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    build_host(force, verbose)
    return LIB


def build_host(force: bool = False, verbose: bool = False) -> Path:
    """_kf_host: recompiled when its source, the C-ABI header or torch changes (a stamp beside the objects says for which it was built)."""
    import torch

    troot = Path(torch.__file__).resolve().parent
    cxx = os.environ.get("CXX", "g++")
    stamp = CSRC / "build" / "kf_host.stamp"
    h = hashlib.sha256(HOST_SRC.read_bytes() + (PKG.parent / "include" / "kf_b200.h").read_bytes())
    h.update(f"{torch.__version__} {sys.version} {cxx}".encode())
    if not force and HOST_LIB.exists() and stamp.exists() and stamp.read_text() == h.hexdigest():
        return HOST_LIB
    cuda = Path(NVCC).resolve().parent.parent
    inc = [sysconfig.get_paths()["include"], troot / "include", troot / "include" / "torch" / "csrc" / "api" / "include", cuda / "include"]
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-I{p}" for p in inc], str(HOST_SRC), "-o", str(HOST_LIB), f"-L{troot / 'lib'}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda",
           "-lc10", "-lc10_cuda", f"-L{PKG}", f"-l:{LIB.name}", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{cxx} failed for {HOST_SRC.name}:\n{r.stdout}\n{r.stderr}")
    if verbose:
        print(r.stderr)
    stamp.write_text(h.hexdigest())
    return HOST_LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))

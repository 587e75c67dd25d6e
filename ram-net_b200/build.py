"""Build libramnet_b200.so (the C-ABI library) in-tree with nvcc for sm_100a, and _host.so (the native host path,
csrc/host/rn_host.cpp: calls from Python arguments to kernel launches) with g++ against the installed torch.

    python ram-net_b200/build.py [--force] [--verbose]

Each csrc/*.cu is compiled to an object file under ram-net_b200/build/ (in parallel) and the
objects are linked into ram-net_b200/ramnet_ops/libramnet_b200.so.  Objects newer than their
sources and headers are reused.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
OBJ = HERE / "build"
LIB = HERE / "ramnet_ops" / "libramnet_b200.so"
HOST_SRC = CSRC / "host" / "rn_host.cpp"
HOST = HERE / "ramnet_ops" / "_host.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(exe).exists():
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build libramnet_b200.so")
    return exe


def _newest(paths) -> float:
    return max(p.stat().st_mtime for p in paths)


def _host_object() -> list[str]:
    """Command that compiles the host module (all but the output path)."""
    import torch
    inc = Path(torch.__file__).resolve().parent / "include"
    cuda = Path(nvcc()).resolve().parent.parent / "include"
    return [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            "-I", str(inc), "-I", str(inc / "torch" / "csrc" / "api" / "include"), "-I", sysconfig.get_paths()["include"],
            "-I", str(cuda), "-c", str(HOST_SRC)]


def _link_host(obj: Path) -> None:
    import torch
    lib = Path(torch.__file__).resolve().parent / "lib"
    cmd = [shutil.which("g++") or "g++", "-shared", "-o", str(HOST), str(obj), "-L", str(LIB.parent), f"-l:{LIB.name}", "-L", str(lib),
           "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10", "-Wl,-rpath,$ORIGIN"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link of {HOST.name} failed:\n{res.stdout}\n{res.stderr}")


def build(force: bool = False, verbose: bool = False) -> Path:
    sources = sorted(CSRC.glob("*.cu"))
    headers = sorted(CSRC.glob("*.cuh")) + [HERE.parent / "include" / "ramnet_b200.h"]
    OBJ.mkdir(exist_ok=True)
    dep_time = _newest(headers)
    jobs = []
    for src in sources:
        obj = OBJ / (src.stem + ".o")
        if force or not obj.exists() or obj.stat().st_mtime < max(src.stat().st_mtime, dep_time):
            jobs.append((src, obj))
    host_obj = OBJ / "rn_host.o"
    host_jobs = []
    if force or not host_obj.exists() or host_obj.stat().st_mtime < max(HOST_SRC.stat().st_mtime, headers[-1].stat().st_mtime):
        host_jobs.append((HOST_SRC, host_obj))

    def compile_one(job):
        src, obj = job
        cmd = [*_host_object(), "-o", str(obj)] if src == HOST_SRC else [nvcc(), *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
        if verbose and src != HOST_SRC:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"compilation of {src.name} failed:\n{res.stdout}\n{res.stderr}")
        if verbose:
            print(res.stderr)
        return obj

    if jobs or host_jobs:
        with ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as pool:
            list(pool.map(compile_one, jobs + host_jobs))
    objs = [OBJ / (s.stem + ".o") for s in sources]
    if force or jobs or not LIB.exists() or LIB.stat().st_mtime < _newest(objs):
        cmd = [nvcc(), "-shared", "-o", str(LIB), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a",
               "-Xcompiler", "-fPIC", "-lcudart"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    if host_jobs or not HOST.exists():
        _link_host(host_obj)
    return LIB


if __name__ == "__main__":
    lib = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(lib)

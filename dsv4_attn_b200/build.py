#!/usr/bin/env python3
"""Build the two shared objects in-tree: libdsv4_attn.so (the kernels behind their C ABI; plain nvcc, no torch) and
_host.<python>.torch-<version>.so (the Python operator surface's fast path; g++ against torch's headers, hence one
file per version of both).

    python -m dsv4_attn_b200.build            # builds what is out of date
    python -m dsv4_attn_b200.build --ptxas-v  # also prints registers / spills / shared memory

The recipe of the first mirrors the reference project's standalone build
(hca/compile.py:68-83): one nvcc call, sm_100a only, a shared object that is
loaded with ctypes.
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
from pathlib import Path

HERE = Path(__file__).resolve().parent
SOURCE = HERE / "csrc" / "api.cu"
OUT = HERE / "libdsv4_attn.so"
HEADER = HERE.parent / "include" / "dsv4_attn.h"
HOST_SOURCE = HERE / "csrc" / "host.cpp"
DEPS = [p for p in sorted((HERE / "csrc").glob("*")) if p != HOST_SOURCE] + [HEADER]


def needs_build(out: Path = OUT, deps=tuple(DEPS)) -> bool:
    if not out.exists():
        return True
    t = out.stat().st_mtime
    return any(p.stat().st_mtime > t for p in deps)


def host_path() -> Path:
    """The native module's file: it is compiled against torch's C++ classes and Python's ABI, so it serves the versions it was built for only."""
    import torch
    return HERE / f"_host.{sys.implementation.cache_tag}.torch-{torch.__version__}.so"


def build_host(force: bool = False, quiet: bool = False) -> Path:
    out = host_path()
    if not force and not needs_build(out, (HOST_SOURCE, HEADER)):
        return out
    import sysconfig

    import torch
    root = Path(torch.__file__).resolve().parent
    nvcc = shutil.which(os.environ.get("NVCC", "nvcc")) or "/usr/local/cuda/bin/nvcc"
    cuda = Path(nvcc).resolve().parent.parent
    cmd = [os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f"-I{sysconfig.get_paths()['include']}", "-isystem", str(root / "include"), "-isystem", str(root / "include" / "torch" / "csrc" / "api" / "include"),
           "-isystem", str(cuda / "include"), "-o", str(out), str(HOST_SOURCE), f"-L{root / 'lib'}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda",
           "-ltorch", "-ltorch_python"]
    if not quiet:
        print(" ".join(cmd), flush=True)
    subprocess.run(cmd, check=True)
    return out


def build(force: bool = False, ptxas_v: bool = False, quiet: bool = False) -> Path:
    build_host(force=force and not ptxas_v, quiet=quiet)
    if not force and not needs_build():
        return OUT
    nvcc = shutil.which(os.environ.get("NVCC", "nvcc")) or "/usr/local/cuda/bin/nvcc"
    cmd = [nvcc, "-std=c++17", "-O3", "-lineinfo",
           "-gencode", "arch=compute_100a,code=sm_100a",
           "-shared", "-Xcompiler", "-fPIC",
           "-o", str(OUT), str(SOURCE)]
    if ptxas_v:
        cmd[1:1] = ["-Xptxas", "-v"]
    if not quiet:
        print(" ".join(cmd), flush=True)
    subprocess.run(cmd, check=True)
    return OUT


def main() -> int:
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--ptxas-v", action="store_true")
    args = ap.parse_args()
    build(force=args.force or args.ptxas_v, ptxas_v=args.ptxas_v)
    print(OUT)
    return 0


if __name__ == "__main__":
    sys.exit(main())

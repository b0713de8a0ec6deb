"""Builds librt_b200.so (the C-ABI kernel library, nvcc for sm_100a) and _rt_torch.so (the
tensor-level entry points over it, g++ against the installed torch) in-tree.

Usage: python -m racetrack_b200.build [--force] [--verbose]

Both are written next to this file under ``lib/``; they are the only binaries the package
loads. nvcc cross-compiles, so no GPU is needed to build.
"""
from __future__ import annotations

import hashlib
import importlib.util
import os
import subprocess
import sys
import sysconfig
from pathlib import Path

from . import _lib

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_DIR = PKG_DIR / "lib"
LIB_PATH = LIB_DIR / "librt_b200.so"
TORCH_PATH = _lib.TORCH_PATH
STAMP = LIB_DIR / "librt_b200.stamp"

# Flags per source. The element-wise kernels are built without FMA contraction so
# that fp32 expressions round exactly like the op-by-op torch path they replace.
SOURCES = {
    "rt_api.cu": [],
    "rt_norm.cu": ["-fmad=false"],
    "rt_act.cu": ["-fmad=false"],
    "rt_moe.cu": ["-fmad=false"],
    "rt_gemm.cu": [],
    "rt_attn.cu": [],
    "rt_peer.cu": ["-fmad=false"],
}

COMMON = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    cuda_home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cand = Path(cuda_home) / "bin" / "nvcc"
    return str(cand) if cand.exists() else "nvcc"


def _fingerprint() -> str:
    h = hashlib.sha256()
    for path in sorted(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.cpp"))
                       + [PKG_DIR.parent / "include" / "rt_b200.h", Path(__file__)]):
        h.update(path.name.encode())
        h.update(path.read_bytes())
    # _rt_torch.so is compiled against the installed torch and the running Python
    h.update(_lib.torch_abi().encode())
    h.update(" ".join(_torch_command()).encode())
    return h.hexdigest()


def _torch_command() -> list[str]:
    torch_dir = Path(importlib.util.find_spec("torch").origin).parent
    cuda_home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    includes = [torch_dir / "include", torch_dir / "include/torch/csrc/api/include",
                sysconfig.get_paths()["include"], f"{cuda_home}/include"]
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wall",
            "-DTORCH_EXTENSION_NAME=_rt_torch", *[f"-isystem{d}" for d in includes],
            str(CSRC / "rt_torch.cpp"), "-o", str(TORCH_PATH), f"-L{torch_dir / 'lib'}",
            "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python",
            f"-Wl,-rpath,{torch_dir / 'lib'}"]


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every source and link the shared libraries; no-op when up to date."""
    LIB_DIR.mkdir(exist_ok=True)
    fp = _fingerprint()
    if not force and LIB_PATH.exists() and TORCH_PATH.exists() and STAMP.exists() and STAMP.read_text() == fp:
        return LIB_PATH
    nvcc = _nvcc()
    objs = []
    procs = []
    for src, extra in SOURCES.items():
        obj = LIB_DIR / (Path(src).stem + ".o")
        cmd = [nvcc, *COMMON, *extra, "-c", str(CSRC / src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
            print(" ".join(cmd), flush=True)
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(str(obj))
    procs.append(("rt_torch.cpp", subprocess.Popen(_torch_command(), stdout=subprocess.PIPE,
                                                   stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, proc in procs:
        out, _ = proc.communicate()
        if proc.returncode != 0:
            failed = True
            sys.stderr.write(f"compilation of {src} failed:\n{out}\n")
        elif verbose or out.strip():
            sys.stderr.write(out)
    if failed:
        raise RuntimeError("librt_b200 build failed")
    link = [nvcc, "-shared", "-o", str(LIB_PATH), *objs, "-lcudart"]
    subprocess.run(link, check=True)
    _lib.TORCH_STAMP.write_text(_lib.torch_abi())
    STAMP.write_text(fp)
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)

"""Compile the CUDA sources of libnnb200 for sm_100a with nvcc, in-tree.

    python -m nnops_b200.build [--force] [--verbose]

Output: nnops_b200/lib/libnnb200.so, and torch_front.*.so, the tensor front end's compiled half for this interpreter's
torch, where there is one with CUDA and a C++ compiler (git-ignored; shipped to GPU machines as built files).
nvcc cross-compiles without a GPU.  -fmad=false keeps every f32 multiply and add separately
rounded unless a kernel asks for an fma explicitly -- the int8 requantisation must match the
CPU arithmetic bit for bit.
"""
from __future__ import annotations

import os
import re
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB_DIR = PKG / "lib"
LIB = LIB_DIR / "libnnb200.so"
FRONT_SRC = PKG / "host" / "torch_front.cpp"
NVCC = os.environ.get("NNB200_NVCC", "/usr/local/cuda/bin/nvcc")
CXX = os.environ.get("NNB200_CXX", "g++")

SOURCES = ["capi.cu", "gemm_i8_umma.cu", "gemm_i8_umma_batched.cu", "i8_realign.cu", "gemm_i8_simt.cu", "gemm_i8_decode.cu", "gemm_i8_skinny.cu", "q4_1_gemv.cu", "q4_1_gemv_mma.cu", "q4_1_gemv_dsq.cu", "q4_1_gemm_umma.cu", "q4_1_rows_umma.cu", "gemm_f16_umma.cu", "shard_gather.cu", "quant_linear.cu", "prepack.cu", "static_scratch.cu", "mma_peak.cu", "conv2d_i8.cu"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-std=c++17", "-O3", "-lineinfo", "-fmad=false",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "--expt-relaxed-constexpr",
]


def _headers(src: Path, seen: set[Path] | None = None) -> set[Path]:
    """The project headers ``src`` includes, directly or through others."""
    seen = set() if seen is None else seen
    for name in re.findall(r'^#include "([^"]+)"', src.read_text(), re.M):
        h = (src.parent / name).resolve()
        if h.exists() and h not in seen:
            seen.add(h)
            _headers(h, seen)
    return seen


def _stale(out: Path, deps: list[Path]) -> bool:
    if not out.exists():
        return True
    t = out.stat().st_mtime
    return any(d.stat().st_mtime > t for d in deps if d.exists())


def build_front(force: bool = False) -> Path | None:
    """host/torch_front.cpp against this interpreter's torch; None, with nothing built, where that has no CUDA or there
    is no compiler.  ops.py does without it."""
    try:
        import torch
    except ImportError:
        return None
    if torch.version.cuda is None or shutil.which(CXX) is None:
        return None
    from . import capi
    out = capi.front_path()
    if force or _stale(out, [FRONT_SRC, PKG.parent / "include" / "nnb200.h"]):
        root = Path(torch.__file__).resolve().parent
        include = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", sysconfig.get_paths()["include"],
                   Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"]
        r = subprocess.run([CXX, "-std=c++17", "-O2", "-fPIC", "-shared", "-fvisibility=hidden",
                            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-isystem{i}" for i in include),
                            str(FRONT_SRC), "-o", str(out), f"-L{root / 'lib'}", f"-Wl,-rpath,{root / 'lib'}", "-ltorch_python",
                            "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10"], capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"{CXX} failed on {FRONT_SRC.name}:\n{r.stdout}\n{r.stderr}")
    return out


def build(force: bool = False, verbose: bool = False) -> Path:
    LIB_DIR.mkdir(exist_ok=True)
    obj_dir = LIB_DIR / "obj"
    obj_dir.mkdir(exist_ok=True)
    flags = list(NVCC_FLAGS) + (["-Xptxas", "-v"] if verbose else [])

    def compile_one(name: str) -> Path:
        src = CSRC / name
        obj = obj_dir / (name + ".o")
        if force or _stale(obj, [src, *_headers(src)]):
            r = subprocess.run([NVCC, *flags, "-c", str(src), "-o", str(obj)], capture_output=True, text=True)
            if r.returncode != 0:
                raise RuntimeError(f"nvcc failed on {name}:\n{r.stdout}\n{r.stderr}")
            if verbose:
                print(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=len(SOURCES)) as ex:
        objs = list(ex.map(compile_one, SOURCES))
    if force or _stale(LIB, objs):
        r = subprocess.run([NVCC, "-shared", "-o", str(LIB), *map(str, objs)],
                           capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    build_front(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))

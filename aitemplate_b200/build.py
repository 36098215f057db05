"""In-tree build of libb200ait.so (hand-written sm_100a kernels + the C-ABI runtime).

The reference compiles a fresh shared library per model with nvcc
(python/aitemplate/backend/builder.py:398-527). Here every kernel is prebuilt once into one
library that all models share; `python -m aitemplate_b200.build` rebuilds it.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys
from pathlib import Path
from typing import List

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_DIR = PKG_DIR / "lib"
LIB_PATH = LIB_DIR / "libb200ait.so"
OBJ_DIR = PKG_DIR / "build"

NVCC_FLAGS = [
    "-std=c++17",
    "-O3",
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "--use_fast_math",
    "-Xcompiler",
    "-fPIC,-fvisibility=hidden",
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; libb200ait.so cannot be built")
    return cand


def sources() -> List[Path]:
    return sorted(CSRC.glob("*.cu"))


def _headers_mtime() -> float:
    hdrs = list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + list((PKG_DIR.parent / "include").glob("*.h"))
    return max((h.stat().st_mtime for h in hdrs), default=0.0)


def _compile_one(src: Path, verbose: bool) -> Path:
    obj = OBJ_DIR / (src.stem + ".o")
    newest = max(src.stat().st_mtime, _headers_mtime())
    if obj.exists() and obj.stat().st_mtime >= newest:
        return obj
    cmd = [_nvcc(), *NVCC_FLAGS, "-I", str(PKG_DIR.parent / "include"), "-c", str(src), "-o", str(obj)]
    if verbose:
        print(" ".join(cmd), flush=True)
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stdout}\n{res.stderr}")
    return obj


def build_calls(force: bool = False, verbose: bool = False) -> Path:
    """Compiles csrc/torch_calls.cpp, the host path of the eager calls, against the installed torch. The file's name says which
    build of torch and of Python it is for."""
    import sysconfig

    import torch

    from . import _lib

    out = _lib.calls_path()
    src, root = CSRC / "torch_calls.cpp", Path(torch.__file__).resolve().parent
    newest = max(src.stat().st_mtime, _headers_mtime())
    if not force and out.exists() and out.stat().st_mtime >= newest:
        return out
    cuda = Path(_nvcc()).resolve().parent.parent
    includes = [PKG_DIR.parent / "include", root / "include", root / "include/torch/csrc/api/include", cuda / "include",
                Path(sysconfig.get_paths()["include"])]
    cmd = ["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    cmd += [a for i in includes for a in ("-I", str(i))]
    cmd += [str(src), "-o", str(out), "-L", str(root / "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    if verbose:
        print(" ".join(cmd), flush=True)
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed for {src.name}:\n{res.stdout}\n{res.stderr}")
    return out


def build_library(force: bool = False, verbose: bool = False) -> Path:
    """Compiles csrc/*.cu for sm_100a and links lib/libb200ait.so, and builds the host path of the eager calls beside
    it. Returns the library's path."""
    LIB_DIR.mkdir(exist_ok=True)
    OBJ_DIR.mkdir(exist_ok=True)
    if force:
        for o in OBJ_DIR.glob("*.o"):
            o.unlink()
    srcs = sources()
    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs) + 1)) as ex:
        calls = ex.submit(build_calls, force, verbose)
        objs = list(ex.map(lambda s: _compile_one(s, verbose), srcs))
    newest_obj = max(o.stat().st_mtime for o in objs)
    if force or not LIB_PATH.exists() or LIB_PATH.stat().st_mtime < newest_obj:
        cmd = [_nvcc(), "-shared", "-o", str(LIB_PATH), *map(str, objs)]
        if verbose:
            print(" ".join(cmd), flush=True)
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    calls.result()  # (the library is complete without it)
    return LIB_PATH


if __name__ == "__main__":
    path = build_library(force="--force" in sys.argv, verbose=True)
    print(path)

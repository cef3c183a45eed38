"""Builds ``zenith_b200/lib/libzenith_b200.so`` from ``zenith_b200/csrc/*.cu`` with nvcc for sm_100a, and
``zenith_b200/lib/_native.so`` (the native host path of the operators, against torch's headers) with g++.

The library links against the static CUDA runtime only, so it loads on a machine without a
driver (compute entry points then return an error status).  Objects are rebuilt only when a
source or header under ``csrc/`` or ``include/`` is newer than the object.

    python -m zenith_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
INCLUDE = PKG.parent / "include"
LIB_DIR = PKG / "lib"
OBJ_DIR = LIB_DIR / "obj"
LIB_PATH = LIB_DIR / "libzenith_b200.so"
NATIVE_SRC = CSRC / "host" / "native_ops.cpp"
NATIVE_PATH = LIB_DIR / "_native.so"

NVCC_FLAGS = [
    "-std=c++17",
    "-O3",
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-Xcompiler",
    "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found (set NVCC or put it on PATH)")


def _newest_header() -> float:
    hdrs = list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + list(INCLUDE.glob("*.h"))
    return max(p.stat().st_mtime for p in hdrs)


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every kernel translation unit and link the shared library; returns its path."""
    nvcc = _nvcc()
    OBJ_DIR.mkdir(parents=True, exist_ok=True)
    sources = sorted(CSRC.glob("*.cu"))
    if not sources:
        raise RuntimeError(f"no .cu sources under {CSRC}")
    hdr_time = max(_newest_header(), Path(__file__).stat().st_mtime)

    def compile_one(src: Path) -> tuple[Path, bool]:
        obj = OBJ_DIR / (src.stem + ".o")
        if not force and obj.exists() and obj.stat().st_mtime > max(src.stat().st_mtime, hdr_time):
            return obj, False
        cmd = [nvcc, *NVCC_FLAGS, "-I", str(INCLUDE), "-c", str(src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
            print(" ".join(cmd), flush=True)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose and r.stderr:
            print(r.stderr, file=sys.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stdout}\n{r.stderr}")
        return obj, True

    with ThreadPoolExecutor(max_workers=min(8, len(sources))) as ex:
        results = list(ex.map(compile_one, sources))
    objs = [o for o, _ in results]
    rebuilt = any(changed for _, changed in results)
    if rebuilt or force or not LIB_PATH.exists():
        cmd = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(LIB_PATH), *map(str, objs)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    _build_native(force)
    return LIB_PATH


def _build_native(force: bool) -> None:
    """The Python module: linked against the library beside it (found through ``$ORIGIN``) and torch's libraries, which
    the interpreter has loaded by the time it imports this one."""
    newest = max(p.stat().st_mtime for p in (NATIVE_SRC, INCLUDE / "zenith_b200.h", Path(__file__)))
    if not force and NATIVE_PATH.exists() and NATIVE_PATH.stat().st_mtime > newest:
        return
    import torch

    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parent.parent
    inc = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", sysconfig.get_paths()["include"],
           cuda / "include"]
    cmd = ["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-fvisibility=hidden", "-DUSE_CUDA",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[f"-I{i}" for i in inc], str(NATIVE_SRC),
           f"-L{LIB_DIR}", "-lzenith_b200", "-Wl,-rpath,$ORIGIN", f"-L{root / 'lib'}", "-ltorch_python", "-ltorch_cuda",
           "-ltorch_cpu", "-lc10_cuda", "-lc10", "-o", str(NATIVE_PATH)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for {NATIVE_SRC.name}:\n{r.stdout}\n{r.stderr}")


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)

"""Builds the native library in-tree with nvcc (sm_100a only).

The kernels are plain CUDA C++ with ``extern "C"`` entry points and no PyTorch
headers, so each translation unit compiles in seconds and the result is one
shared object, ``kempnerforge_b200/lib/libkfb200.so``, loaded through ctypes.

One host file reads Python modules and tensors (``csrc/steps.cpp``) and is built
against the headers of Python and PyTorch into a CPython module beside it.  It serves
only the versions that it was built for, so its name holds them; the library serves any.
"""

from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import torch

PKG_ROOT = Path(__file__).resolve().parent.parent
REPO_ROOT = PKG_ROOT.parent
CSRC = REPO_ROOT / "csrc"
LIB_DIR = PKG_ROOT / "lib"
LIB_PATH = LIB_DIR / "libkfb200.so"
STEPS_PATH = LIB_DIR / f"kf_steps.{sysconfig.get_config_var('SOABI')}.torch-{torch.__version__}.so"

NVCC_FLAGS = [
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-O3",
    "-std=c++17",
    "--use_fast_math",
    "-Xcompiler",
    "-fPIC",
    "-Xptxas",
    "-v",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found; set NVCC or add it to PATH")


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _fingerprint() -> str:
    h = hashlib.sha256()
    for f in sorted(f for kind in ("*.cu", "*.cuh", "*.h", "*.cpp") for f in CSRC.glob(kind)):
        h.update(f.name.encode())
        h.update(f.read_bytes())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def _build_steps() -> None:
    """``csrc/steps.cpp`` -> a CPython module."""
    root = Path(torch.__file__).parent
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I", str(root / "include"), "-I", str(root / "include" / "torch" / "csrc" / "api" / "include"),
           "-I", sysconfig.get_paths()["include"], str(CSRC / "steps.cpp"), "-o", str(STEPS_PATH),
           "-L", str(root / "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed for steps.cpp:\n{res.stderr[-4000:]}")


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every ``csrc/*.cu`` and link them into the shared library (no-op when up to date)."""
    LIB_DIR.mkdir(exist_ok=True)
    stamp = LIB_DIR / "build.stamp"
    fp = _fingerprint()
    if not force and LIB_PATH.exists() and STEPS_PATH.exists() and stamp.exists() and stamp.read_text() == fp:
        return LIB_PATH
    nvcc = _nvcc()
    obj_dir = REPO_ROOT / "build" / "obj"
    obj_dir.mkdir(parents=True, exist_ok=True)
    log_dir = REPO_ROOT / "build" / "ptxas"
    log_dir.mkdir(parents=True, exist_ok=True)

    def compile_one(src: Path) -> Path:
        obj = obj_dir / (src.stem + ".o")
        cmd = [nvcc, *NVCC_FLAGS, "-I", str(CSRC), "-c", str(src), "-o", str(obj)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        (log_dir / (src.stem + ".log")).write_text(res.stderr)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stderr[-4000:]}")
        if verbose:
            print(res.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(sources())))) as pool:
        steps = pool.submit(_build_steps)
        objs = list(pool.map(compile_one, sources()))
        steps.result()
    link = [nvcc, "-shared", "-o", str(LIB_PATH), *map(str, objs),]
    res = subprocess.run(link, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stderr[-4000:]}")
    stamp.write_text(fp)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force=True, verbose=True))

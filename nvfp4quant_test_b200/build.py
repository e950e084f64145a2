"""Compile libnvfp4_b200.so (sm_100a only, nvcc) and the compiled half of the entry points (_native, g++) in-tree.

  python -m nvfp4quant_test_b200.build [--force]
"""
from __future__ import annotations

import os
import pathlib
import shutil
import subprocess
import sys
import sysconfig

PKG = pathlib.Path(__file__).resolve().parent
CSRC = PKG / "csrc"
INCLUDE = PKG.parent / "include"
LIB = PKG / "libnvfp4_b200.so"
NATIVE_SRC = CSRC / "host" / "native.cpp"
NATIVE = PKG / ("_native" + sysconfig.get_config_var("EXT_SUFFIX"))

SOURCES = ["quant.cu", "global_scale.cu", "global_scale_static.cu", "importance.cu", "dequant.cu", "gemm.cu", "status.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-fmad=false",  # every fused multiply-add in the kernels is written explicitly
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not pathlib.Path(cand).exists():
        raise RuntimeError("nvcc not found; set NVCC or install the CUDA toolkit")
    return cand


def _stale() -> bool:
    if not LIB.exists():
        return True
    t = LIB.stat().st_mtime
    deps = [CSRC / s for s in SOURCES] + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.inc")) + list(INCLUDE.glob("*.h"))
    return any(d.stat().st_mtime > t for d in deps if d.exists())


def build(force: bool = False, verbose: bool = False) -> pathlib.Path:
    """Build the shared library and the extension module, each if it is missing or older than its sources."""
    if force or _stale():
        _build_lib(verbose)
    deps = [NATIVE_SRC, *INCLUDE.glob("*.h")]
    if force or not NATIVE.exists() or any(d.stat().st_mtime > NATIVE.stat().st_mtime for d in deps):
        _build_native()
    return LIB


def _build_native() -> None:
    """The CPython module that checks arguments, allocates and launches; linked against the library beside it."""
    import torch

    torch_dir = pathlib.Path(torch.__file__).resolve().parent
    cuda = pathlib.Path(_nvcc()).resolve().parents[1]
    includes = [INCLUDE, sysconfig.get_paths()["include"], torch_dir / "include",
                torch_dir / "include" / "torch" / "csrc" / "api" / "include", cuda / "include"]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", *[f"-I{d}" for d in includes],
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", str(NATIVE_SRC), "-o", str(NATIVE),
           f"-L{PKG}", f"-L{torch_dir / 'lib'}", f"-L{cuda / 'lib64'}", "-lnvfp4_b200", "-lc10", "-lc10_cuda", "-ltorch_cpu",
           "-ltorch_cuda", "-ltorch_python", "-lcudart", "-Wl,-rpath,$ORIGIN"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("g++ failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)


def _build_lib(verbose: bool) -> pathlib.Path:
    srcs = [str(CSRC / s) for s in SOURCES if (CSRC / s).exists()]
    extra = os.environ.get("NVFP4_EXTRA_NVCC_FLAGS", "").split()   # e.g. -DNVFP4_QUANT_MIN_BLOCKS=6 for experiments
    cmd = [_nvcc(), *NVCC_FLAGS, *extra, f"-I{INCLUDE}", f"-I{CSRC}", "-shared", "-o", str(LIB), *srcs]
    if verbose:
        cmd.insert(1, "-Xptxas=-v")
    env = dict(os.environ)
    # nvcc picks its host compiler itself; a CC/CXX meant for another toolchain would only mislead it
    env.pop("CC", None)
    env.pop("CXX", None)
    res = subprocess.run(cmd, capture_output=True, text=True, env=env)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
    if verbose:
        print(res.stderr)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))

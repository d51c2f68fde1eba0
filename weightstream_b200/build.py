"""Builds ``libws_tp.so`` (the C-ABI CUDA library, nvcc for sm_100a) and ``_ws_torch.so`` (its front end
for torch tensors, g++) in-tree."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libws_tp.so")
TORCH_EXT = os.path.join(HERE, "_ws_torch.so")
SOURCES = ["ws_api.cu", "ws_bootstrap.cu"]
HEADERS = ["ws_device.cuh", "ws_fp8_kernel.cuh", "ws_fp8_gemv_kernel.cuh", "ws_fp8_bs_kernel.cuh", "ws_fp8_tile_kernel.cuh", "ws_moe_kernel.cuh", "ws_moe_gemv_kernel.cuh", "ws_moe_bs_kernel.cuh", "ws_misc_kernels.cuh",
           os.path.join("..", "..", "include", "ws_tp.h")]


def nvcc_path() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; the CUDA library cannot be built")


def _older(target: str, sources) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in sources if os.path.exists(d))


def is_stale() -> bool:
    return _older(LIB, [os.path.join(CSRC, f) for f in SOURCES + HEADERS]) or _torch_ext_is_stale()


def _abi() -> str:
    """What the front end's binary interface depends on, kept beside it: it loads with no other Python or torch."""
    from importlib.metadata import version
    return f"python {sys.version_info[0]}.{sys.version_info[1]} torch {version('torch')}"


def _torch_ext_is_stale() -> bool:
    if _older(TORCH_EXT, [os.path.join(CSRC, "ws_torch.cpp"), os.path.join(CSRC, HEADERS[-1])]):
        return True
    try:
        with open(TORCH_EXT + ".abi") as f:
            return f.read() != _abi()
    except OSError:
        return True


def _run(cmd, verbose: bool) -> None:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose:
        sys.stderr.write(res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"{os.path.basename(cmd[0])} failed:\n" + res.stdout + res.stderr)


def build(force: bool = False, verbose: bool = False) -> str:
    if force or _older(LIB, [os.path.join(CSRC, f) for f in SOURCES + HEADERS]):
        _run([nvcc_path(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
              "-shared", "-Xcompiler", "-fPIC", "-Xptxas", "-v" if verbose else "-O3",
              "-o", LIB] + [os.path.join(CSRC, s) for s in SOURCES] + ["-lcudart"], verbose)
    if force or _torch_ext_is_stale():
        import sysconfig

        import torch
        t = os.path.dirname(torch.__file__)
        cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc_path()))), "include")
        _run([os.environ.get("CXX") or "g++", "-O2", "-std=c++17", "-shared", "-fPIC",
              "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI,
              "-I" + os.path.join(t, "include"), "-I" + os.path.join(t, "include", "torch", "csrc", "api", "include"),
              "-I" + cuda, "-I" + sysconfig.get_paths()["include"], os.path.join(CSRC, "ws_torch.cpp"), "-o", TORCH_EXT,
              "-L" + HERE, "-lws_tp", "-L" + os.path.join(t, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python",
              "-Wl,-rpath,$ORIGIN"], verbose)
        with open(TORCH_EXT + ".abi", "w") as f:
            f.write(_abi())
    return LIB


if __name__ == "__main__":
    print(build(force=True, verbose="-v" in sys.argv))

"""Build step: compile the CUDA sources under ``csrc/`` into ``lib/libhbq_b200.so`` and the
torch-facing entry points (``csrc/host.cpp``) into ``lib/hbq_host.so``.

The library targets sm_100a only and depends on nothing but the CUDA runtime, so it
cross-compiles on a machine without a GPU; the module is built against the installed torch (and is left out where that
has no CUDA) and rebuilt when torch or Python has changed::

    python -m hbq_b200.build
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libhbq_b200.so")
HOST_PATH = os.path.join(LIB_DIR, "hbq_host.so")
HOST_SOURCE = os.path.join(CSRC, "host.cpp")
SOURCES = ["api.cu", "quantize.cu", "quantize_lut.cu", "quantize_tab.cu", "quantize_extra.cu", "dequantize.cu", "gemm_simt.cu", "gemm_tc.cu", "gemm_packed.cu", "gemm_static.cu", "moe.cu", "rope.cu"]
HEADERS = [os.path.join(CSRC, "common.cuh"), os.path.join(CSRC, "quantize_dev.cuh"), os.path.join(CSRC, "vcache_dev.cuh"), os.path.join(CSRC, "quantize_tab.cuh"), os.path.join(CSRC, "tc_dev.cuh"), os.path.join(HERE, "..", "include", "hbq_b200.h")]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-shared", "--threads", "4"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; it is needed to build libhbq_b200.so")


def _older(path: str, deps) -> bool:
    return not os.path.exists(path) or any(os.path.getmtime(d) > os.path.getmtime(path) for d in deps)


def is_stale() -> bool:
    return _older(LIB_PATH, [os.path.join(CSRC, s) for s in SOURCES] + HEADERS)


def host_tag():
    """What ``hbq_host.so`` is compiled for -- torch, its CUDA and C++ ABI, this Python; None where torch has no CUDA."""
    import torch
    if torch.version.cuda is None:
        return None
    return (f"hbq_host for torch {torch.__version__} cuda {torch.version.cuda} cxx11abi {int(torch._C._GLIBCXX_USE_CXX11_ABI)} "
            f"python {sysconfig.get_config_var('SOABI')}")


def host_matches(path=None) -> bool:
    """The module at ``path`` (the built one) carries this process's tag."""
    tag, path = host_tag(), path or HOST_PATH
    if tag is None or not os.path.exists(path):
        return False
    with open(path, "rb") as f:
        return tag.encode() + b"\0" in f.read()


def host_is_stale() -> bool:
    return host_tag() is not None and (_older(HOST_PATH, [HOST_SOURCE, HEADERS[-1]]) or not host_matches())


def _host_command(out: str):
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            f'-DHBQ_HOST_TAG="{host_tag()}"', "-o", out, HOST_SOURCE, *["-I" + i for i in inc],
            "-L" + os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"]


def build_library(force: bool = False, verbose: bool = False) -> str:
    """Compile what is missing or out of date; return the library's path."""
    host = None
    os.makedirs(LIB_DIR, exist_ok=True)
    made = f"{HOST_PATH}.{os.getpid()}"                                  # renamed when complete: the old one may be loaded
    if host_tag() is not None and (force or host_is_stale()):
        env = {k: v for k, v in os.environ.items() if k not in ("CC", "CXX")}
        host = subprocess.Popen(_host_command(made), env=env)           # beside nvcc
    try:
        if force or is_stale():
            _build_cuda(verbose)
    finally:
        if host is not None:
            if host.wait() != 0:
                raise RuntimeError("building hbq_host.so failed")
            os.replace(made, HOST_PATH)
    return LIB_PATH


def _build_cuda(verbose: bool) -> None:
    cmd = [_nvcc(), *NVCC_FLAGS, "-o", LIB_PATH, *[os.path.join(CSRC, s) for s in SOURCES]]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
        print(" ".join(cmd))
    env = dict(os.environ)
    # nvcc's host compiler: the image exports a CC wrapper that is not a full gcc install
    env.pop("CC", None)
    env.pop("CXX", None)
    subprocess.check_call(cmd, env=env)


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))

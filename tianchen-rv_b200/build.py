"""Build recipe for the provider's native code (sm_100a only, in-tree outputs).

``build_library()`` has the Makefile compile ``csrc/*.cu`` into ``libtcrv_cuda.so`` next to this file
with nvcc; it needs no GPU (nvcc cross-compiles).  ``build_torch_calls()`` compiles
``csrc/torch_calls.cpp``, the package's native call path, into ``_tcrv_torch.<Python ABI>.torch-<version>.so``
beside it with the host compiler.  Run as a script to force a rebuild.
"""
from __future__ import annotations

import contextlib
import fcntl
import glob
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libtcrv_cuda.so")


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: the provider's CUDA library cannot be built")
    return exe


def _stale() -> bool:
    if not os.path.exists(LIB):
        return True
    built = os.path.getmtime(LIB)
    deps = [p for kind in ("*.cu", "*.cuh", "*.h") for p in glob.glob(os.path.join(CSRC, kind))]
    deps += glob.glob(os.path.join(ROOT, "include", "*.h")) + glob.glob(os.path.join(HERE, "Makefile"))
    return any(os.path.getmtime(p) > built for p in deps)


@contextlib.contextmanager
def _one_builder():
    """Processes that build at the same time share the objects: one after another."""
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    with open(os.path.join(HERE, "build", "lock"), "w") as f:
        fcntl.flock(f, fcntl.LOCK_EX)
        yield


def build_library(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return LIB
    cmd = ["make", "-C", HERE, f"-j{os.cpu_count()}", f"NVCC={_nvcc()}", "library"]
    if force:
        cmd.insert(1, "-B")
    if verbose:
        cmd.append("NVCCEXTRA=-Xptxas=-v")
        print(" ".join(cmd), file=sys.stderr)
    else:
        cmd.insert(1, "-s")
    with _one_builder():
        if force or _stale():  # (another process may have built it meanwhile)
            subprocess.run(cmd, check=True)
    return LIB


def torch_calls_path() -> str:
    """Where the native call path is for this interpreter and this torch.  It is compiled against
    CPython's and torch's C++ headers, so a build for others must not be loaded: the name tells them apart."""
    import torch

    return os.path.join(HERE, f"_tcrv_torch.{sysconfig.get_config_var('SOABI')}.torch-{torch.__version__}.so")


def build_torch_calls(force: bool = False) -> str:
    """The Python calls' native half; needs the C-ABI library (it links against it)."""
    import torch

    out = torch_calls_path()
    source = os.path.join(CSRC, "torch_calls.cpp")
    deps = [source, os.path.join(ROOT, "include", "tcrv_cuda.h"), os.path.abspath(__file__)]
    if not force and os.path.exists(out) and all(os.path.getmtime(d) <= os.path.getmtime(out) for d in deps):
        return out
    torch_dir = os.path.dirname(torch.__file__)
    torch_lib = os.path.join(torch_dir, "lib")
    cuda_include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "include")
    subprocess.run([
        os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
        f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
        "-I", os.path.join(ROOT, "include"), "-I", sysconfig.get_paths()["include"],
        "-isystem", os.path.join(torch_dir, "include"), "-isystem", os.path.join(torch_dir, "include/torch/csrc/api/include"),
        "-isystem", cuda_include, "-o", out, source,
        "-L", HERE, "-ltcrv_cuda", "-L", torch_lib, "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda",
        "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{torch_lib}",
    ], check=True)
    return out


if __name__ == "__main__":
    import importlib.util

    print(build_library(force=True, verbose="-v" in sys.argv))
    if importlib.util.find_spec("torch") is not None:  # the C library needs none
        print(build_torch_calls(force=True))

"""Builds libtritt_sm100.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a, and the host extension _host with g++.

    python flash-3-way-attention_b200/build.py [--force] [--verbose]

Every ``csrc/*.cu`` is compiled to an object file under ``csrc/build/`` (skipped when
the object is newer than the source and every header), then linked into
``flash_trittention/libtritt_sm100.so`` with the CUDA runtime linked statically, so
that the library does not depend on which CUDA runtime the host process loaded.  The host extension is for one version of
Python (its file's suffix) and of PyTorch (``csrc/build/host.txt`` and the module say which); without g++ or Python's headers the
library is built alone, and the package does with Python what the extension would do.
"""
from __future__ import annotations

import concurrent.futures as cf
import glob
import os
import shutil
import subprocess
import sys
import sysconfig
import warnings

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(CSRC, "build")
LIB = os.path.join(HERE, "flash_trittention", "libtritt_sm100.so")
HOST_SRC = os.path.join(CSRC, "host", "tritt_host.cpp")
HOST = os.path.join(HERE, "flash_trittention", "_host" + sysconfig.get_config_var("EXT_SUFFIX"))
HOST_STAMP = os.path.join(OBJ, "host.txt")
ABI_HEADER = os.path.join(HERE, "..", "include", "tritt.h")

NVCC_FLAGS = [
    "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
    "-Xcompiler", "-fPIC", "--use_fast_math", "-Xptxas", "-v",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _host_recipe() -> list:
    """The command that builds the host extension, PyTorch's version in it.  Raises where something it needs is not installed."""
    import torch

    if shutil.which("g++") is None:
        raise RuntimeError("g++ not found")
    root, include = os.path.dirname(torch.__file__), sysconfig.get_paths()["include"]
    if not os.path.exists(os.path.join(include, "Python.h")):
        raise RuntimeError(f"no Python.h in {include}")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "include")
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            f'-DTRITT_TORCH_VERSION="{torch.__version__}"', f"-I{root}/include", f"-I{root}/include/torch/csrc/api/include", f"-I{cuda}",
            f"-I{include}", f"-I{os.path.dirname(ABI_HEADER)}", HOST_SRC, "-o", HOST, f"-L{root}/lib", "-lc10", "-lc10_cuda", "-ltorch_cpu",
            "-ltorch", "-ltorch_python"]


def host_is_current(recipe: list) -> bool:
    """Whether the extension there is was built by this recipe (this PyTorch and Python) from these files."""
    if not os.path.exists(HOST) or not os.path.exists(HOST_STAMP) or open(HOST_STAMP).read() != "\n".join(recipe):
        return False
    return os.path.getmtime(HOST) > max(os.path.getmtime(HOST_SRC), os.path.getmtime(ABI_HEADER))


def build_host(force: bool = False) -> str:
    """The extension module that makes a call's checks and allocations natively (a host program against PyTorch's headers)."""
    recipe = _host_recipe()
    if not force and host_is_current(recipe):
        return HOST
    r = subprocess.run(recipe, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for {HOST_SRC}:\n{r.stdout}\n{r.stderr}")
    with open(HOST_STAMP, "w") as f:
        f.write("\n".join(recipe))
    return HOST


def build_host_if_possible(force: bool = False) -> None:
    try:
        build_host(force)
    except RuntimeError as e:
        warnings.warn(f"the host extension was not built, short calls will take twice as long: {e}")


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    nvcc = _nvcc()
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    hdrs = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    newest_hdr = max(os.path.getmtime(h) for h in hdrs)

    def compile_one(src):
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        if (not force and os.path.exists(obj) and os.path.getmtime(obj) > max(os.path.getmtime(src), newest_hdr)):
            return obj, ""
        cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
        return obj, r.stderr

    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        results = list(ex.map(compile_one, srcs))
    objs = [o for o, _ in results]
    if verbose:
        for _, log in results:
            if log:
                print(log)
    if force or not os.path.exists(LIB) or any(os.path.getmtime(o) > os.path.getmtime(LIB) for o in objs):
        cmd = [nvcc, "-shared", "-cudart", "static", "-gencode", "arch=compute_100a,code=sm_100a",
               "-Xcompiler", "-fPIC", "-o", LIB, *objs]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    build_host_if_possible(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))

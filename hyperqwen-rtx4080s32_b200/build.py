"""Build the CUDA library in-tree for sm_100a, hyperqwen-rtx4080s32_b200/libgq_b200.so, and the Python extension that
calls it without ctypes, hyperqwen-rtx4080s32_b200/_gq_torch.so.

nvcc cross-compiles without a GPU.  The format tables are generated first from the installed gguf
package (csrc/gen_tables.py).  `python -m hyperqwen_rtx4080s32_b200.build` or build() from Python.
"""
from __future__ import annotations

import os
import subprocess
import sys

_HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(_HERE, "csrc")
LIB = os.path.join(_HERE, "libgq_b200.so")
EXT = os.path.join(_HERE, "_gq_torch.so")
SOURCES = ["gq_b200.cu"]
EXT_SOURCE = os.path.join(CSRC, "gq_torch.cpp")
EXT_STAMP = os.path.join(CSRC, "_generated", "gq_torch.stamp")     # what the extension was compiled against
HEADERS = sorted(f for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))) + [os.path.join("..", "..", "include", "gq_b200.h")]
NVCC_FLAGS = ["-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "--expt-relaxed-constexpr", "-diag-suppress", "177",
              "-shared", "-Xcompiler", "-fPIC"]


def _newest(paths):
    return max(os.path.getmtime(p) for p in paths if os.path.exists(p))


def build(force: bool = False, verbose: bool = False) -> str:
    sys.path.insert(0, CSRC)
    try:
        import gen_tables
    finally:
        sys.path.pop(0)
    table_h = gen_tables.generate()
    srcs = [os.path.join(CSRC, s) for s in SOURCES]
    deps = srcs + [os.path.join(CSRC, h) for h in HEADERS] + [table_h]
    if force or not os.path.exists(LIB) or os.path.getmtime(LIB) < _newest(deps):
        _build_lib(srcs, verbose)
    if force or not _ext_current():
        _build_ext()
    return LIB


def _ext_tag() -> str:
    """The binary interfaces the extension is compiled against: torch's C++ classes and this Python's."""
    import sysconfig

    import torch

    return f"torch {torch.__version__} cxx11abi {int(torch._C._GLIBCXX_USE_CXX11_ABI)} python {sysconfig.get_config_var('SOABI')}"


def _ext_current() -> bool:
    if not os.path.exists(EXT) or os.path.getmtime(EXT) < _newest([EXT_SOURCE, os.path.join(CSRC, HEADERS[-1])]):
        return False
    try:
        with open(EXT_STAMP) as f:
            return f.read() == _ext_tag()
    except OSError:
        return False


def _build_lib(srcs, verbose: bool) -> None:
    nvcc = os.environ.get("NVCC") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else "nvcc")
    cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB] + srcs
    subprocess.check_call(cmd, cwd=CSRC)


def _build_ext() -> None:
    import sysconfig

    import torch

    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME") or "/usr/local/cuda"
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include"),
           sysconfig.get_paths()["include"]]
    cmd = [os.environ.get("CXX") or "g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] + ["-I" + d for d in inc]
    cmd += [EXT_SOURCE, "-o", EXT, "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10",
            "-L" + _HERE, "-lgq_b200", "-Wl,-rpath,$ORIGIN"]
    subprocess.check_call(cmd, cwd=CSRC)
    with open(EXT_STAMP, "w") as f:
        f.write(_ext_tag())


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))

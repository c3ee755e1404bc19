"""Builds libcombskv.so (the C-ABI library) in-tree with nvcc for sm_100a."""
from __future__ import annotations

import importlib.machinery
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libcombskv.so")
LIB_MEASURE = os.path.join(HERE, "libcombskv_measure.so")  # -DCBKV_MEASURE: per-role timers, switches read from CBKV_DEBUG
SOURCES = ["manager.cpp", "sessions.cpp", "kernels.cu", "prefill_tc.cu", "chunk_pair.cu", "rope.cu", "kvquant.cu", "api.cu", "noalloc.cu"]
HEADERS = ["manager.hpp", "kernels.hpp", "pdl.cuh", "tile.cuh", "tc.cuh", "rope.cuh", "q8_unpack.cuh", os.path.join("..", "..", "include", "combs_kv.h")]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-shared", "-cudart", "static", "-ldl",
]


PYCALL_SOURCE = os.path.join(CSRC, "pycall.cpp")


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def needs_build(lib: str = LIB) -> bool:
    if not os.path.exists(lib):
        return True
    t = os.path.getmtime(lib)
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS] + [os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False, measure: bool = False) -> str:
    """The product library, or (measure=True) the measurement flavour: the same sources with
    -DCBKV_MEASURE, which adds timers and phase switches the product build does not contain."""
    lib = LIB_MEASURE if measure else LIB
    if not force and not needs_build(lib):
        return lib
    cmd = [_nvcc(), *NVCC_FLAGS, *( ["-DCBKV_MEASURE"] if measure else []), "-ccbin", "/usr/bin/g++",
           *[os.path.join(CSRC, f) for f in SOURCES], "-o", lib]
    if verbose:
        cmd.insert(1, "-Xptxas=-v")
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + r.stdout + r.stderr)
    if verbose:
        sys.stderr.write(r.stderr)
    return lib


def pycall_path() -> str:
    """The Python mirror's hot calls (csrc/pycall.cpp).  The file is bound to torch's C++ and to CPython's binary interface, so
    its name carries both versions: another torch or Python finds no file of its own instead of one that does not load."""
    import torch
    return os.path.join(HERE, f"_pycall.torch-{torch.__version__}{importlib.machinery.EXTENSION_SUFFIXES[0]}")


def build_pycall(force: bool = False) -> str:
    """Needs torch and Python's headers, unlike the library; without the file the same calls go through ctypes."""
    path = pycall_path()
    if not force and os.path.exists(path) and os.path.getmtime(path) >= os.path.getmtime(PYCALL_SOURCE):
        return path
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    cmd = ["/usr/bin/g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-w", "-I" + sysconfig.get_paths()["include"], "-I" + os.path.join(root, "include"),
           "-I" + os.path.join(root, "include", "torch", "csrc", "api", "include"), "-I/usr/local/cuda/include", PYCALL_SOURCE,
           "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-o", path]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("g++ failed:\n" + r.stdout + r.stderr)
    return path


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv, measure="--measure" in sys.argv))
    try:
        print(build_pycall(force="--force" in sys.argv))
    except (ImportError, RuntimeError) as e:
        print(f"not built, the Python calls go through ctypes: {e}")

"""Build recipe of the CUDA library (one nvcc call, sm_100a only) and of the label collation (a CPython extension,
one call of the C compiler), output next to the sources.

    python -m elmo_b200.build            # builds elmo_b200/_build/libelmo_xmc.so and _collate.so if stale
"""
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT_DIR = os.path.join(HERE, "_build")
LIB = os.path.join(OUT_DIR, "libelmo_xmc.so")
SOURCES = ["xmc_lib.cu"]
HEADERS = ["ptx.cuh", "numerics.cuh", "gemm_engine.cuh", "xmc_policies.cuh", "aux_kernels.cuh", "gradx_kernel.cuh", "slim_step.cuh",
           os.path.join("..", "..", "include", "elmo_xmc.h")]


def _stale():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS] + [os.path.abspath(__file__)]
    return any(os.path.exists(d) and os.path.getmtime(d) > t for d in deps)


COLLATE_SRC = os.path.join(CSRC, "collate.c")
COLLATE = os.path.join(OUT_DIR, "_collate.so")


def build_collate(force=False):
    """Compile the label collation against this interpreter's headers; returns its path, or None where the
    headers or a C compiler are missing (the glue then collates with numpy)."""
    if not force and os.path.exists(COLLATE) and os.path.getmtime(COLLATE) >= os.path.getmtime(COLLATE_SRC):
        return COLLATE
    include = sysconfig.get_path("include")
    if not os.path.exists(os.path.join(include, "Python.h")):
        return None
    os.makedirs(OUT_DIR, exist_ok=True)
    try:
        res = subprocess.run([os.environ.get("CC", "gcc"), "-O2", "-shared", "-fPIC", "-I", include, "-o", COLLATE, COLLATE_SRC],
                             capture_output=True, text=True)
    except OSError:
        return None
    if res.returncode != 0:
        raise RuntimeError("the C compiler failed:\n" + res.stdout + res.stderr)
    return COLLATE


def build(force=False, verbose=False):
    """Compile the library for sm_100a (nvcc cross-compiles without a GPU). Returns the .so path."""
    build_collate(force)
    if not force and not _stale():
        return LIB
    os.makedirs(OUT_DIR, exist_ok=True)
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    cmd = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
           "-Xcompiler", "-fPIC", "-shared", "-cudart", "static",
           "-Xptxas", "-v" if verbose else "-warn-spills",
           "-o", LIB] + [os.path.join(CSRC, s) for s in SOURCES]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    if verbose:
        print(res.stderr)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))

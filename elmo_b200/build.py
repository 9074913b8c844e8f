"""Build recipe of the CUDA library (one nvcc call, sm_100a only) and of the label collation (a CPython extension,
one call of the C compiler), output next to the sources.

    python -m elmo_b200.build            # builds elmo_b200/_build/libelmo_xmc.so and _collate.*.so if stale
"""
import os
import subprocess
import sys
import sysconfig
import warnings

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
# the extension belongs to one interpreter version: its tag is part of the name
COLLATE = os.path.join(OUT_DIR, "_collate" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))


def built_collate():
    """Path of the label collation if it is built and not older than its source, else None."""
    try:
        return COLLATE if os.path.getmtime(COLLATE) >= os.path.getmtime(COLLATE_SRC) else None
    except OSError:
        return None


def build_collate(force=False):
    """Compile the label collation against this interpreter's headers; returns its path, or None, with a warning,
    where that cannot be done (the glue then collates with numpy).  Other processes find the whole file or none:
    it is written under a name of this process's own and renamed."""
    if not force and built_collate():
        return COLLATE
    tmp = "%s.%d.tmp" % (COLLATE, os.getpid())
    try:
        os.makedirs(OUT_DIR, exist_ok=True)
        res = subprocess.run([os.environ.get("CC", "gcc"), "-O2", "-shared", "-fPIC", "-I", sysconfig.get_path("include"),
                              "-o", tmp, COLLATE_SRC], capture_output=True, text=True)
        if res.returncode != 0:
            raise OSError("the C compiler failed:\n" + res.stdout + res.stderr)
        os.replace(tmp, COLLATE)
    except OSError as e:
        warnings.warn("label collation not built, numpy does it: %s" % e)
        if os.path.exists(tmp):
            os.unlink(tmp)
        return None
    return COLLATE


def build(force=False, verbose=False):
    """Compile the library for sm_100a (nvcc cross-compiles without a GPU). Returns the .so path.  What the compiler has
    to say about kernels that spill registers goes to stderr."""
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
    if res.stderr.strip():                    # the resource usage of every kernel, or the spill warnings
        print(res.stderr, file=sys.stdout if verbose else sys.stderr)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))

"""Builds build/libnanoserve.so (the C-ABI library) from nanoserve_b200/csrc with nvcc for sm_100a.

The library keeps the reference project's name and location (build/libnanoserve.so relative to the
repository root, cf. the reference's python/nanoserve/ops.py:12) so a caller that loads the reference
library by path loads this one unchanged.
"""
import glob
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "nanoserve_b200", "csrc")
LIB_DIR = os.path.join(ROOT, "build")
LIB_PATH = os.path.join(LIB_DIR, "libnanoserve.so")
CALL_SRC = os.path.join(CSRC, "binding.cpp")
CALL_PATH = os.path.join(LIB_DIR, "nanoserve_call.so")  # Python extension: the host side of an eager call

NVCC_FLAGS = [
    "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
    "-Xcompiler", "-fPIC", "-shared", "--threads", "0",
]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale():
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + \
        glob.glob(os.path.join(ROOT, "include", "*.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def built_for() -> str:
    """What the Python extension is bound to: torch's C++ classes and the interpreter."""
    import torch
    return f"torch {torch.__version__} {sys.implementation.cache_tag}"


def call_matches(path: str) -> bool:
    """Whether the extension at `path` was built for this torch and this interpreter (a note beside it says for which)."""
    try:
        with open(path + ".built_for") as f:
            return f.read() == built_for()
    except OSError:
        return False


def build_call(force: bool = False) -> str:
    """Compile the Python extension (host code on torch's C++ objects; no CUDA sources) if its source is newer or it was built
    for another torch or Python."""
    if not force and os.path.exists(CALL_PATH) and call_matches(CALL_PATH) and \
            os.path.getmtime(CALL_PATH) >= os.path.getmtime(CALL_SRC):
        return CALL_PATH
    import sysconfig
    import torch
    os.makedirs(LIB_DIR, exist_ok=True)
    t = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    include = [os.path.join(t, "include"), os.path.join(t, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    lib = os.path.join(t, "lib")
    part = f"{CALL_PATH}.{os.getpid()}"  # whole before it has its name: another process may be loading it
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-I{i}" for i in include], CALL_SRC, "-o", part, f"-L{lib}", f"-Wl,-rpath,{lib}",
           "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    res = subprocess.run(cmd, cwd=ROOT, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("g++ failed building nanoserve_call.so")
    if os.path.exists(CALL_PATH + ".built_for"):
        os.remove(CALL_PATH + ".built_for")  # never a note beside an extension that it is not about
    os.replace(part, CALL_PATH)
    with open(part, "w") as f:
        f.write(built_for())
    os.replace(part, CALL_PATH + ".built_for")
    return CALL_PATH


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile the library and the Python extension if any source is newer. Returns the library path.

    The library needs nvcc alone.  Where the extension cannot be built as well (no g++, no headers of Python or torch) eager
    calls go through ctypes."""
    _build_library(force, verbose)
    try:
        build_call(force)
    except Exception as e:  # whatever is missing: the library is complete without it
        sys.stderr.write(f"nanoserve_call.so was not built, eager calls go through ctypes: {e!r}\n")
    return LIB_PATH


def _build_library(force, verbose):
    if not force and not _stale():
        return
    os.makedirs(LIB_DIR, exist_ok=True)
    nvcc = os.environ.get("NVCC", "nvcc")
    cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB_PATH] + sources()
    env = dict(os.environ)
    # nvcc picks the host compiler from PATH; a CC/CXX override in the environment is not used
    res = subprocess.run(cmd, cwd=ROOT, env=env, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("nvcc failed building libnanoserve.so")
    if verbose:
        sys.stderr.write(res.stderr)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))

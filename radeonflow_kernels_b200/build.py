"""In-tree build of librf_b200.so (sm_100a only) with nvcc, and of the CPython extension _host.so with the host compiler.

    python -m radeonflow_kernels_b200.build [--force] [--verbose]

The shared library is written next to this file so that it travels with the
source tree; nothing is installed into site-packages and there is no JIT cache.
"""
import glob
import os
import shutil
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "librf_b200.so")
HOST_SRC = os.path.join(CSRC, "host_path.cpp")
HOST_PATH = os.path.join(PKG_DIR, "_host.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-shared",
]


def _nvcc() -> str:
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; librf_b200.so cannot be built")


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale() -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(CSRC, "*.cuh"))
    deps += glob.glob(os.path.join(CSRC, "*.inc"))
    deps.append(os.path.join(os.path.dirname(PKG_DIR), "include", "rf_b200.h"))
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def build_host(force: bool = False) -> str:
    """The extension is bound to the interpreter that builds it."""
    if not force and os.path.exists(HOST_PATH) and os.path.getmtime(HOST_PATH) >= os.path.getmtime(HOST_SRC):
        return HOST_PATH
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + sysconfig.get_paths()["include"],
           "-o", HOST_PATH, HOST_SRC]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("building _host.so failed")
    return HOST_PATH


def build(force: bool = False, verbose: bool = False) -> str:
    build_host(force)
    if not force and not _stale():
        return LIB_PATH
    cmd = [_nvcc()] + NVCC_FLAGS
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += ["-o", LIB_PATH] + sources() + ["-lcudart"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed building librf_b200.so")
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))

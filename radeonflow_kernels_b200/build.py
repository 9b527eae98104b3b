"""In-tree build of librf_b200.so (sm_100a only) with nvcc, and of the CPython extension _host with the host compiler.

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
HOST_PATH = os.path.join(PKG_DIR, "_host" + sysconfig.get_config_var("EXT_SUFFIX"))

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


def _compile(cmd, path, verbose=False):
    """Runs cmd, which ends in `-o`, its output and more; the file appears whole, for other processes that build or load it."""
    tmp = f"{path}.{os.getpid()}.tmp"
    try:
        res = subprocess.run([tmp if c == path else c for c in cmd], capture_output=True, text=True)
        if verbose or res.returncode != 0:
            sys.stderr.write(res.stdout + res.stderr)
        if res.returncode != 0:
            raise RuntimeError(f"building {os.path.basename(path)} failed")
        os.replace(tmp, path)
    finally:
        if os.path.exists(tmp):
            os.remove(tmp)


def build_host(force: bool = False) -> str:
    """The extension is bound to the interpreter that builds it, and its name says to which."""
    if not force and os.path.exists(HOST_PATH) and os.path.getmtime(HOST_PATH) >= os.path.getmtime(HOST_SRC):
        return HOST_PATH
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + sysconfig.get_paths()["include"],
           "-o", HOST_PATH, HOST_SRC]
    _compile(cmd, HOST_PATH)
    return HOST_PATH


def build(force: bool = False, verbose: bool = False) -> str:
    """Path of the library.  The extension is built too where that is possible; without it the Python code does its work."""
    if force or _stale():
        cmd = [_nvcc()] + NVCC_FLAGS
        if verbose:
            cmd += ["-Xptxas", "-v"]
        _compile(cmd + ["-o", LIB_PATH] + sources() + ["-lcudart"], LIB_PATH, verbose)
    try:
        build_host(force)
    except (RuntimeError, OSError) as e:        # no host compiler, or no Python headers
        sys.stderr.write(f"{e}: the Python boundary runs without its extension\n")
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))

"""Build recipe for the native library: every .cu under csrc/ is compiled for
sm_100a with nvcc into one shared object, ``q8_kernels_b200/libq8k_b200.so``,
which exports the C ABI declared in ``include/q8_kernels_b200.h``; ``csrc/host.cpp`` becomes the CPython extension
``q8_kernels_b200/_host.<interpreter>.so`` over it, against the headers and libraries of the installed torch.  Its
name carries the interpreter's ABI tag, so another Python does not load it.

Run ``python q8_kernels_b200/build.py`` (add ``--force`` to rebuild, ``-v`` for
ptxas resource usage).  nvcc cross-compiles without a GPU present.  A program that calls the C ABI needs
neither torch nor Python headers: ``--library-only``, or a machine without torch, builds the library alone.
"""
from __future__ import annotations

import argparse
import importlib.util
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
OBJ_DIR = os.path.join(PKG_DIR, "build")
LIB_PATH = os.path.join(PKG_DIR, "libq8k_b200.so")
HOST_PATH = os.path.join(PKG_DIR, "_host" + sysconfig.get_config_var("EXT_SUFFIX"))
HOST_KEY = os.path.join(OBJ_DIR, os.path.basename(HOST_PATH) + ".key")     # what the extension was built against

SOURCES = ["capi.cu", "rowwise.cu", "hadamard.cu", "gemm.cu", "gemm_pair.cu", "gemm_split.cu", "attention.cu"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _build_host(force: bool) -> None:
    src = os.path.join(CSRC, "host.cpp")
    header = os.path.join(PKG_DIR, "..", "include", "q8_kernels_b200.h")
    torch = importlib.util.find_spec("torch")
    if torch is None:
        sys.stderr.write(f"torch is not installed: {os.path.basename(LIB_PATH)} is built, the extension of the Python package is not\n")
        return
    untagged = os.path.join(PKG_DIR, "_host.so")                 # of a build before the names were tagged
    if os.path.exists(untagged) and untagged != HOST_PATH:
        os.remove(untagged)
    torch_dir = os.path.dirname(torch.origin)
    with open(os.path.join(torch_dir, "version.py")) as f:
        key = torch_dir + "\n" + f.read()                        # another torch needs another build
    if not (force or _stale(HOST_PATH, [src, header]) or not os.path.exists(HOST_KEY) or open(HOST_KEY).read() != key):
        return
    abi = subprocess.run([sys.executable, "-c", "import torch; print(int(torch.compiled_with_cxx11_abi()))"],
                         capture_output=True, text=True, cwd=OBJ_DIR)
    if abi.returncode != 0:
        sys.stderr.write(abi.stderr)
        raise RuntimeError("torch does not import")
    inc = [sysconfig.get_paths()["include"], os.path.join(torch_dir, "include"),
           os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"),
           os.path.join(os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda", "include")]
    cmd = (["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-D_GLIBCXX_USE_CXX11_ABI=" + abi.stdout.strip()]
           + ["-I" + d for d in inc]
           + [src, "-o", HOST_PATH, "-L" + os.path.join(torch_dir, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python",
              "-L" + PKG_DIR, "-l:libq8k_b200.so", "-Wl,-rpath,$ORIGIN"])
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("g++ failed on host.cpp")
    with open(HOST_KEY, "w") as f:
        f.write(key)


def build(force: bool = False, verbose: bool = False, library_only: bool = False) -> str:
    """Compile the library if any source is newer than it, and the Python package's extension over it unless
    ``library_only``; return the library's path."""
    os.makedirs(OBJ_DIR, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(PKG_DIR, "..", "include", "q8_kernels_b200.h"))
    nvcc = _nvcc()
    flags = list(NVCC_FLAGS) + (["-Xptxas", "-v"] if verbose else [])

    def compile_one(src: str) -> str:
        obj = os.path.join(OBJ_DIR, src.replace(".cu", ".o"))
        path = os.path.join(CSRC, src)
        if force or _stale(obj, [path] + headers):
            cmd = [nvcc] + flags + ["-c", path, "-o", obj]
            res = subprocess.run(cmd, capture_output=True, text=True)
            if verbose or res.returncode != 0:
                sys.stderr.write(res.stdout + res.stderr)
            if res.returncode != 0:
                raise RuntimeError(f"nvcc failed on {src}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(SOURCES))) as pool:
        objs = list(pool.map(compile_one, SOURCES))
    if force or _stale(LIB_PATH, objs):
        cmd = [nvcc, "-shared", "-o", LIB_PATH] + objs + ["-lcudart"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            sys.stderr.write(res.stdout + res.stderr)
            raise RuntimeError("link failed")
    if not library_only:
        _build_host(force)
    return LIB_PATH


if __name__ == "__main__":
    ap = argparse.ArgumentParser(description=__doc__)
    ap.add_argument("--force", action="store_true")
    ap.add_argument("-v", "--verbose", action="store_true")
    ap.add_argument("--library-only", action="store_true", help="the C ABI without the Python package's extension")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose, library_only=a.library_only))

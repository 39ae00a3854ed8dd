"""Builds lib/libixk.so from csrc/*.cu with nvcc for sm_100a (cross-compiles without a GPU), and lib/ixk_calls-*.so, the
Python package's native calls, from csrc/py_calls.cc with the host compiler against the installed torch.

Run as a script (python build.py [--force] [--verbose]) or call build().
Objects go to build/ next to this file; both folders are git-ignored build products.
"""
from __future__ import annotations

import concurrent.futures
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
OBJ_DIR = os.path.join(HERE, "build")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libixk.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
    "-I", INCLUDE, "-I", CSRC,
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; libixk.so cannot be built")
    return exe


def _newest(paths) -> float:
    return max(os.path.getmtime(p) for p in paths)


def build(force: bool = False, verbose: bool = False, ptxas_info: bool = False) -> str:
    """Compile and link; returns the path of the shared library."""
    sources = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    headers.append(os.path.join(INCLUDE, "ixk.h"))
    os.makedirs(OBJ_DIR, exist_ok=True)
    os.makedirs(LIB_DIR, exist_ok=True)
    nvcc = _nvcc()
    hdr_time = _newest(headers + [os.path.abspath(__file__)])

    def compile_one(src: str):
        src_path = os.path.join(CSRC, src)
        obj = os.path.join(OBJ_DIR, src[:-3] + ".o")
        if (not force and os.path.exists(obj)
                and os.path.getmtime(obj) > max(os.path.getmtime(src_path), hdr_time)):
            return obj, ""
        cmd = [nvcc, *NVCC_FLAGS, "-c", src_path, "-o", obj]
        if ptxas_info:
            cmd[1:1] = ["-Xptxas", "-v"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
        return obj, r.stderr

    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(sources))) as pool:
        results = list(pool.map(compile_one, sources))
    objs = [o for o, _ in results]
    if verbose or ptxas_info:
        for (_, log), src in zip(results, sources):
            if log.strip():
                print(f"--- {src}\n{log}", file=sys.stderr)
    if force or not os.path.exists(LIB_PATH) or os.path.getmtime(LIB_PATH) < _newest(objs):
        cmd = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB_PATH, *objs,
               "-cudart", "static"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    try:
        build_calls(force)
    except (ImportError, OSError, RuntimeError) as e:      # (the library and the Python package work without)
        print(f"native calls not built, the package's calls go through Python: {e}", file=sys.stderr)
    return LIB_PATH


def calls_path(lib_dir: str = LIB_DIR) -> str:
    """Where the native calls for this interpreter and torch are.  They use torch's C++ classes, whose layout is each
    version's own: one built against another is another file, which nobody loads."""
    import torch
    made_for = f"torch{torch.__version__}-cxx{int(torch._C._GLIBCXX_USE_CXX11_ABI)}"
    return os.path.join(lib_dir, f"ixk_calls-{made_for}{sysconfig.get_config_var('EXT_SUFFIX')}")


def build_calls(force: bool = False) -> str:
    import torch
    path = calls_path()
    source = os.path.join(CSRC, "py_calls.cc")
    inputs = [source, os.path.join(INCLUDE, "ixk.h"), os.path.abspath(__file__)]
    if not force and os.path.exists(path) and os.path.getmtime(path) > _newest(inputs):
        return path
    home = os.path.dirname(torch.__file__)
    cuda_include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "include")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I", INCLUDE, "-I", os.path.join(home, "include"), "-I", os.path.join(home, "include", "torch", "csrc", "api", "include"),
           "-I", sysconfig.get_paths()["include"], "-I", cuda_include, source, "-o", path,
           "-L", os.path.join(home, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10_cuda", "-lc10"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed on py_calls.cc:\n{r.stdout}\n{r.stderr}")
    return path


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv,
                 ptxas_info="--ptxas" in sys.argv)
    print(path)

"""Build the CUDA library in-tree for sm_100a only.

    python -m gdn_qsa_sm80_b200.build [--force] [--verbose]

Compiles every ``csrc/*.cu`` with nvcc (``-gencode arch=compute_100a,code=sm_100a -lineinfo``)
and links ``lib/libgdn_chunk_sm100.so`` next to this file, and the native front end of the Python
wrapper (``csrc/gdn_frontend.cpp``, a CPython extension) as ``lib/_gdn_frontend.so`` beside it.  nvcc cross-compiles, so no GPU is
needed to build.  There is no other architecture, no JIT cache and no fallback target.
"""

from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libgdn_chunk_sm100.so")
FRONTEND_PATH = os.path.join(LIB_DIR, "_gdn_frontend.so")
OBJ_DIR = os.path.join(HERE, "build")
TORCH_STAMP = os.path.join(OBJ_DIR, "frontend_torch_version")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC or add it to PATH)")


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _deps_mtime() -> float:
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    files.append(os.path.join(os.path.dirname(HERE), "include", "gdn_chunk_sm100.h"))
    files.append(os.path.abspath(__file__))
    return max(os.path.getmtime(f) for f in files)


def _torch_version() -> str:
    import importlib.metadata
    return importlib.metadata.version("torch")


def needs_build() -> bool:
    if any(not os.path.exists(p) or os.path.getmtime(p) < _deps_mtime() for p in (LIB_PATH, FRONTEND_PATH)):
        return True
    try:    # the front end links torch's libraries
        with open(TORCH_STAMP) as f:
            return f.read() != _torch_version()
    except OSError:
        return True


def _build_frontend() -> None:
    import sysconfig
    import torch
    torch_dir = os.path.dirname(torch.__file__)
    torch_lib = os.path.join(torch_dir, "lib")
    include = [os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-I{d}" for d in include], os.path.join(CSRC, "gdn_frontend.cpp"), "-o", FRONTEND_PATH,
           f"-L{LIB_DIR}", "-lgdn_chunk_sm100", f"-L{torch_lib}", "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda",
           "-ltorch_python", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("g++ failed on gdn_frontend.cpp")
    with open(TORCH_STAMP, "w") as f:
        f.write(_torch_version())


def build(force: bool = False, verbose: bool = False, diagnostics: bool | None = None) -> str:
    """diagnostics (default: environment variable GDN_BUILD_DIAGNOSTICS=1) compiles the kernels' cycle accounting in
    (-DGDN_DIAGNOSTICS); a production build carries none of it."""
    if diagnostics is None:
        diagnostics = os.environ.get("GDN_BUILD_DIAGNOSTICS", "0") == "1"
    if not force and not needs_build() and not diagnostics:
        return LIB_PATH
    nvcc = _nvcc()
    os.makedirs(LIB_DIR, exist_ok=True)
    os.makedirs(OBJ_DIR, exist_ok=True)
    extra = ["-Xptxas", "-v"] if verbose else []
    if diagnostics:
        extra.append("-DGDN_DIAGNOSTICS")

    def compile_one(src):
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        cmd = [nvcc, *NVCC_FLAGS, *extra, "-c", src, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        return src, obj, r

    with ThreadPoolExecutor(max_workers=4) as ex:
        results = list(ex.map(compile_one, sources()))
    objs = []
    for src, obj, r in results:
        if verbose or r.returncode != 0:
            sys.stderr.write(f"--- {os.path.basename(src)}\n{r.stdout}{r.stderr}\n")
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}")
        objs.append(obj)
    link = [nvcc, "-shared", "-o", LIB_PATH, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
    r = subprocess.run(link, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("link failed")
    _build_frontend()
    return LIB_PATH


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true", help="print ptxas register / shared-memory usage")
    ap.add_argument("--diagnostics", action="store_true", help="compile the kernels' cycle accounting in")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose, diagnostics=a.diagnostics or None))

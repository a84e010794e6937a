"""Build the C-ABI shared library (lib/libck_b200.so) from csrc/*.cu for sm_100a, and the Python
wrappers' native half (lib/_ck_host.so) from csrc/host against the installed torch's headers (without
those, or a C++ compiler for them, the library alone).

    python comfy-kitchen_b200/build.py [--force] [--verbose]

nvcc cross-compiles without a GPU.  The library links the CUDA runtime
statically and resolves the one driver entry point it needs (tensor-map
encoding) at run time, so it loads on machines without a driver too.
"""
from __future__ import annotations

import argparse
import glob
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libck_b200.so")
OBJ_DIR = os.path.join(HERE, "build")
HOST_SRC = os.path.join(CSRC, "host", "ck_host.cpp")
HOST_PATH = os.path.join(LIB_DIR, "_ck_host.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC",
    "-Xcompiler", "-fvisibility=hidden",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC)")


def _sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_host(force: bool = False, verbose: bool = False) -> str:
    """The extension module that backends/cuda calls for plain eager calls (torch is found, not imported)."""
    os.makedirs(LIB_DIR, exist_ok=True)
    torch = importlib.util.find_spec("torch")
    if torch is None:
        raise RuntimeError("torch is not installed")
    torch_dir = list(torch.submodule_search_locations)[0]
    if not force and not _stale(HOST_PATH, [HOST_SRC, os.path.join(torch_dir, "version.py")]):
        return HOST_PATH
    include, libs = os.path.join(torch_dir, "include"), os.path.join(torch_dir, "lib")
    cuda_include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "include")
    cmd = [os.environ.get("CXX") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-I" + include,
           "-I" + os.path.join(include, "torch", "csrc", "api", "include"), "-I" + sysconfig.get_paths()["include"], "-I" + cuda_include,
           HOST_SRC, "-o", HOST_PATH, "-L" + libs, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]
    if verbose:
        print(" ".join(cmd), flush=True)
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        print(r.stdout, flush=True)
        raise RuntimeError(f"{cmd[0]} failed on {HOST_SRC}")
    return HOST_PATH


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(LIB_DIR, exist_ok=True)
    os.makedirs(OBJ_DIR, exist_ok=True)
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + \
        glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    nvcc = _nvcc()
    objs = []
    procs = []
    for src in _sources():
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if force or _stale(obj, [src] + headers):
            cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
                print(" ".join(cmd), flush=True)
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            print(out, flush=True)
        if p.returncode != 0:
            print(f"nvcc failed on {src}", file=sys.stderr)
            failed = True
    if failed:
        raise RuntimeError("build failed")
    if force or procs or _stale(LIB_PATH, objs):
        cmd = [nvcc, "-shared", "-o", LIB_PATH, *objs, "-cudart", "static", "-Xcompiler", "-fPIC"]
        if verbose:
            print(" ".join(cmd), flush=True)
        subprocess.run(cmd, check=True)
    try:
        build_host(force, verbose)
    except (OSError, RuntimeError) as e:  # the library is complete without it; an older one might not fit it
        if os.path.exists(HOST_PATH):
            os.remove(HOST_PATH)
        print(f"host extension not built ({e}): the package's calls will go through its Python wrappers", file=sys.stderr)
    return LIB_PATH


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))

"""Builds libdsv3_b200.so (nvcc, sm_100a) and _dsv3_host.so (g++, against torch's headers) in-tree: no JIT cache, no
pip install.

    python deepseek-v3_b200/build.py [--force] [--verbose]
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT_DIR = os.path.join(HERE, "lib")
LIB = os.path.join(OUT_DIR, "libdsv3_b200.so")
HOST_LIB = os.path.join(OUT_DIR, "_dsv3_host.so")     # CPython extension: argument checks, allocation, launch
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
         "-Xcompiler", "-fPIC,-O2,-Wall", "--expt-relaxed-constexpr"]


def sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _newest_input() -> float:
    paths = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(INCLUDE, "dsv3_b200.h"), __file__]
    return max(os.path.getmtime(p) for p in paths)


def _run(cmd, what: str) -> None:
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{what} failed:\n{r.stdout}\n{r.stderr}")


def _torch_dir() -> str:
    import importlib.util
    return os.path.dirname(importlib.util.find_spec("torch").origin)


def compile_host() -> str:
    """host.cpp against torch's and CPython's headers."""
    inc = os.path.join(_torch_dir(), "include")
    obj = os.path.join(OUT_DIR, "host.o")
    _run(["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-Wall", "-D_GLIBCXX_USE_CXX11_ABI=1", "-I", INCLUDE,
          "-isystem", inc, "-isystem", os.path.join(inc, "torch", "csrc", "api", "include"),
          "-isystem", os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include"),
          "-isystem", sysconfig.get_paths()["include"], "-c", os.path.join(CSRC, "host.cpp"), "-o", obj], "g++ for host.cpp")
    return obj


def link_host(obj: str) -> None:
    libs = os.path.join(_torch_dir(), "lib")
    _run(["g++", "-shared", "-o", HOST_LIB, obj, "-L", OUT_DIR, "-l:libdsv3_b200.so", "-L", libs, "-lc10", "-lc10_cuda",
          "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-L", os.path.join(os.path.dirname(os.path.dirname(NVCC)), "lib64"),
          "-l:libcudart.so.12", "-Wl,-rpath,$ORIGIN"], "link of _dsv3_host.so")


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OUT_DIR, exist_ok=True)
    newest = _newest_input()
    if not force and all(os.path.exists(p) and os.path.getmtime(p) >= newest for p in (LIB, HOST_LIB)):
        return LIB
    ccbin = ["-ccbin", "/usr/bin/g++"] if os.path.exists("/usr/bin/g++") else []
    extra = ["-Xptxas", "-v"] if verbose else []

    def compile_one(src: str) -> str:
        obj = os.path.join(OUT_DIR, src[:-3] + ".o")
        cmd = [NVCC, *FLAGS, *ccbin, *extra, "-I", INCLUDE, "-c", os.path.join(CSRC, src), "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(sources()) + 1)) as ex:
        host = ex.submit(compile_host)
        objs = list(ex.map(compile_one, sources()))
        host_obj = host.result()
    cmd = [NVCC, *ccbin, "-shared", "-o", LIB, *objs, "-cudart", "static"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    link_host(host_obj)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))

"""In-tree build of libhtr_b200.so (nvcc, sm_100a only).  `python -m htr_b200.build [-v] [--force]`.

The shared library has no Python or torch dependency: it exports the C interface of include/htr_b200.h
and is loaded with ctypes (htr_b200/_lib.py).  Objects are compiled in parallel, one per source file;
a source is recompiled when it or any header is newer than its object.  Beside it stands the native front of the operators
(csrc/host_binding.cpp -> _host.so, a CPython extension over torch's C++ API), which reaches the library through addresses.
"""
import concurrent.futures
import glob
import os
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(PKG, "build")
LIB = os.path.join(PKG, "libhtr_b200.so")
HOST = os.path.join(PKG, "_host.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
         "-Xptxas", "-v", "-I", os.path.join(ROOT, "include")]


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _compile(src, obj, verbose):
    r = subprocess.run([NVCC, *FLAGS, "-c", src, "-o", obj], capture_output=True, text=True)
    with open(obj + ".log", "w") as f:
        f.write(r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
    if verbose:
        print(r.stderr)
    return obj


def _compile_host(src):
    import torch

    t = os.path.dirname(torch.__file__)
    include = [os.path.join(t, "include"), os.path.join(t, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"],
               os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include")]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-I{d}" for d in include], src, "-o", HOST, "-L" + os.path.join(t, "lib"),
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for {src}:\n{r.stdout}\n{r.stderr}")


def build(force=False, verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(ROOT, "include", "*.h"))
    jobs = []
    for src in sources:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        if force or _stale(obj, [src, *headers]):
            jobs.append((src, obj))
    host_src = os.path.join(CSRC, "host_binding.cpp")
    with concurrent.futures.ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as ex:
        waiting = [ex.submit(_compile_host, host_src)] if force or _stale(HOST, [host_src, os.path.join(ROOT, "include", "htr_b200.h")]) else []
        waiting += [ex.submit(_compile, s, o, verbose) for s, o in jobs]
        for fut in waiting:
            fut.result()
    objs = [os.path.join(OBJ, os.path.basename(s)[:-3] + ".o") for s in sources]
    if force or jobs or _stale(LIB, objs):
        subprocess.run([NVCC, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "static"],
                       check=True)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))

"""Build libqllm2_pam_b200.so in-tree with nvcc for sm_100a, and _host.so (the host runtime, C++ over torch) beside it.

    python -m qllm2_b200.build [--force] [--verbose]

Each .cu under csrc/ is compiled to an object (in parallel) and linked into one shared
library next to this file; each .cpp under csrc/host/ likewise into a Python module that links against it.  Objects are
rebuilt when a source or header is newer.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libqllm2_pam_b200.so")
HOST_SRC = os.path.join(CSRC, "host")
HOST_LIB = os.path.join(HERE, "_host.so")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I", INCLUDE,
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: cannot build libqllm2_pam_b200.so")
    return exe


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _headers_mtime() -> float:
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    return max(os.path.getmtime(h) for h in hs)


def _compile(src: str, verbose: bool) -> str:
    obj = os.path.join(OBJ, src[:-3] + ".o")
    cmd = [_nvcc(), *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
    if verbose:
        sys.stderr.write(r.stderr)
    return obj


def _host_flags():
    import sysconfig

    import torch
    from torch.utils import cpp_extension as ce
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = ce.include_paths() + [os.path.join(cuda, "include"), sysconfig.get_paths()["include"], INCLUDE]
    flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_host",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[x for i in inc for x in ("-isystem" if i != INCLUDE else "-I", i)]]
    libs = [x for p in ce.library_paths() + [os.path.join(cuda, "lib64")] for x in ("-L", p)]
    libs += ["-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-lcudart"]
    return flags, libs


def _compile_host(src: str, flags) -> str:
    obj = os.path.join(OBJ, "host_" + src[:-4] + ".o")
    r = subprocess.run(["g++", *flags, "-c", os.path.join(HOST_SRC, src), "-o", obj], capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for {src}:\n{r.stdout}\n{r.stderr}")
    return obj


def _stale(target: str, parts) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(p) > os.path.getmtime(target) for p in parts)


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    srcs = _sources()
    hm = _headers_mtime()
    todo, objs = [], []
    for s in srcs:
        obj = os.path.join(OBJ, s[:-3] + ".o")
        objs.append(obj)
        newest = max(os.path.getmtime(os.path.join(CSRC, s)), hm)
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < newest:
            todo.append(s)
    host_srcs = sorted(f for f in os.listdir(HOST_SRC) if f.endswith(".cpp"))
    host_hm = max(os.path.getmtime(os.path.join(d, f)) for d in (HOST_SRC, INCLUDE) for f in os.listdir(d) if f.endswith(".h"))
    host_objs = [os.path.join(OBJ, "host_" + s[:-4] + ".o") for s in host_srcs]
    host_todo = [s for s, o in zip(host_srcs, host_objs)
                 if force or not os.path.exists(o) or os.path.getmtime(o) < max(os.path.getmtime(os.path.join(HOST_SRC, s)), host_hm)]
    flags, libs = _host_flags() if host_todo or not os.path.exists(HOST_LIB) else (None, None)
    if todo or host_todo:
        with cf.ThreadPoolExecutor(max_workers=min(len(todo) + len(host_todo), os.cpu_count() or 4)) as ex:
            jobs = [ex.submit(_compile_host, s, flags) for s in host_todo] + [ex.submit(_compile, s, verbose) for s in todo]
            for j in jobs:
                j.result()
    if _stale(LIB, objs):
        cmd = [_nvcc(), "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a",
               "-lcuda"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    if _stale(HOST_LIB, host_objs):
        if libs is None:
            flags, libs = _host_flags()
        cmd = ["g++", "-shared", "-o", HOST_LIB, *host_objs, "-L", HERE, "-lqllm2_pam_b200", "-Wl,-rpath,$ORIGIN", *libs]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return LIB


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)

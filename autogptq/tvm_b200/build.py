"""Ahead-of-time build of ``libb200gptq.so`` (sm_100a only) with nvcc, and of ``_host`` with the host compiler.

The library is plain CUDA C++ behind a C ABI: it links against the CUDA runtime
and nothing else (no torch, no Python headers), and is placed next to this file
so that it travels with the source tree.  ``_host`` is a small CPython module (torch headers) that prepares a
``QuantLinear.forward`` call in native code and calls the library.  ``python -m autogptq.tvm_b200.build``
rebuilds both; :func:`build` is a no-op when they are newer than every source.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.normpath(os.path.join(HERE, "..", "..", "include"))
LIB_NAME = "libb200gptq.so"
LIB_PATH = os.path.join(HERE, LIB_NAME)
HOST_SRC = os.path.join(CSRC, "host", "host_call.cpp")
HOST_PATH = os.path.join(HERE, "_host" + sysconfig.get_config_var("EXT_SUFFIX"))

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "--shared", "-Xcompiler", "-fPIC",
    "-Xcompiler", "-fvisibility=hidden",
    "--expt-relaxed-constexpr",
    "-cudart", "shared",
]


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _deps():
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if os.path.isfile(os.path.join(CSRC, f))]
    deps += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    return deps


def _host_deps():
    return [HOST_SRC] + [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]


def _older(path, deps) -> bool:
    return not os.path.isfile(path) or any(os.path.getmtime(d) > os.path.getmtime(path) for d in deps)


def _host_command(out: str):
    import torch
    root = os.path.dirname(torch.__file__)
    inc = os.path.join(root, "include")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            "-I", inc, "-I", os.path.join(inc, "torch", "csrc", "api", "include"), "-I", sysconfig.get_paths()["include"],
            "-I", os.path.join(cuda, "include"), HOST_SRC, "-o", out, "-L", HERE, f"-l:{LIB_NAME}", "-Wl,-rpath,$ORIGIN",
            "-L", os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]


def is_stale() -> bool:
    return _older(LIB_PATH, _deps()) or _older(HOST_PATH, _host_deps())


def build(force: bool = False, verbose: bool = False, extra_flags=()) -> str:
    """Build if needed.  Safe when several processes (the ranks of one job) import the package at once: the build
    runs under an exclusive file lock, and a process that waited for the lock finds the library fresh and returns."""
    if not force and not is_stale():
        return LIB_PATH
    import fcntl
    obj_dir = os.path.join(HERE, "build")
    os.makedirs(obj_dir, exist_ok=True)
    with open(os.path.join(obj_dir, ".lock"), "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            if not force and not is_stale():
                return LIB_PATH
            return _build_locked(force, verbose, extra_flags)
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)


def _build_locked(force: bool, verbose: bool, extra_flags) -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: libb200gptq.so cannot be built on this machine")
    objs = []
    obj_dir = os.path.join(HERE, "build")
    os.makedirs(obj_dir, exist_ok=True)
    procs = []
    compile_flags = [f for f in NVCC_FLAGS if f != "--shared"]
    for src in sources():
        obj = os.path.join(obj_dir, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if not force and os.path.isfile(obj) and all(os.path.getmtime(d) <= os.path.getmtime(obj) for d in _deps()):
            continue
        cmd = [nvcc, *compile_flags, *extra_flags, "-I", INCLUDE, "-c", src, "-o", obj]
        if verbose:
            print(" ".join(cmd), file=sys.stderr)
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, p in procs:
        out, _ = p.communicate()
        if verbose and out:
            print(out, file=sys.stderr)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{out}")
    tmp = f"{LIB_PATH}.tmp.{os.getpid()}"
    link = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "--shared", "-cudart", "shared",
            "-o", tmp, *objs]
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}")
    os.replace(tmp, LIB_PATH)
    if not force and not _older(HOST_PATH, _host_deps()):
        return LIB_PATH      # (it binds the library at load time: a new library needs no new host module)
    tmp = f"{HOST_PATH}.tmp.{os.getpid()}"
    cmd = _host_command(tmp)
    if verbose:
        print(" ".join(cmd), file=sys.stderr)
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed for {HOST_SRC}:\n{r.stdout}")
    os.replace(tmp, HOST_PATH)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force=("--force" in sys.argv or "--ptxas-v" in sys.argv), verbose=True,
                extra_flags=("-Xptxas", "-v") if "--ptxas-v" in sys.argv else ()))

"""Build, in-tree: libwkv_b200.so (the C-ABI library, sm_100a only, nvcc) and _wkv_native.so (the
PyTorch binding on top of it, g++).

    python -m rwkv_infctx_trainer_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libwkv_b200.so")
STAMP = LIB + ".digest"
SOURCES = ["wkv_api.cu", "wkv4.cu", "wkv4_par.cu", "wkv56_scalar.cu", "wkv56_chunked.cu", "wkv56_chunked_bwd.cu",
           "timemix_fused.cu", "decode.cu"]
NATIVE_NAME = "_wkv_native"
NATIVE = os.path.join(PKG, NATIVE_NAME + ".so")
NATIVE_SOURCES = ["native_ops.cpp", "native_timemix.cpp", "native_blocks.cpp"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "--use_fast_math", "-Xcompiler", "-fPIC"]


def have_nvcc() -> bool:
    return bool(shutil.which("nvcc")) or os.path.exists("/usr/local/cuda/bin/nvcc")


def have_cxx() -> bool:
    return bool(shutil.which("g++"))


def _digest(files, *more: str) -> str:
    """sha256 over the names and contents of the files and over the other strings"""
    h = hashlib.sha256()
    for f in files:
        h.update(os.path.basename(f).encode())
        with open(f, "rb") as fh:
            h.update(fh.read())
    h.update(" ".join(more).encode())
    return h.hexdigest()


def _source_digest() -> str:
    files = [os.path.join(CSRC, f) for f in sorted(os.listdir(CSRC))
             if f.endswith((".cu", ".cuh", ".h")) and not f.startswith("native_")]
    files.append(os.path.join(PKG, "..", "include", "wkv_b200.h"))
    return _digest(files, *NVCC_FLAGS)


def _native_digest() -> str:
    import torch
    files = [os.path.join(CSRC, f) for f in sorted(os.listdir(CSRC)) if f.startswith("native_") or f == "wkv_internal.h"]
    files.append(os.path.join(PKG, "..", "include", "wkv_b200.h"))
    return _digest(files, torch.__version__, sys.version, *NATIVE_FLAGS)


NATIVE_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-Wall", "-Wextra", f"-DTORCH_EXTENSION_NAME={NATIVE_NAME}"]


def native_is_current() -> bool:
    if not os.path.exists(NATIVE) or not os.path.exists(NATIVE + ".digest"):
        return False
    with open(NATIVE + ".digest") as f:
        return f.read().strip() == _native_digest()


def build_native(force: bool = False) -> str:
    """Compile the PyTorch binding against the installed torch; it links to libwkv_b200.so beside it."""
    if not force and native_is_current():
        return NATIVE
    import torch
    from torch.utils import cpp_extension
    # (-isystem: warnings are for this package's own sources)
    incs = [f"-isystem{p}" for p in [*cpp_extension.include_paths(), "/usr/local/cuda/include", sysconfig.get_paths()["include"]]]
    bdir = os.path.join(PKG, "build")
    os.makedirs(bdir, exist_ok=True)
    procs, objs = [], []
    for s in NATIVE_SOURCES:
        obj = os.path.join(bdir, s.replace(".cpp", f".{os.getpid()}.o"))
        cmd = ["g++", *NATIVE_FLAGS, f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *incs, "-c",
               os.path.join(CSRC, s), "-o", obj]
        procs.append((s, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)))
        objs.append(obj)
    for s, p in procs:
        out = p.communicate()[0].decode()
        if p.returncode != 0:
            raise RuntimeError(f"g++ failed on {s}:\n{out}")
        if out:
            print(out, file=sys.stderr)
    tmp = f"{NATIVE}.{os.getpid()}.tmp"
    tlib = os.path.join(os.path.dirname(torch.__file__), "lib")
    subprocess.check_call(["g++", "-shared", "-o", tmp, *objs, f"-L{PKG}", "-l:libwkv_b200.so", f"-L{tlib}", "-lc10", "-lc10_cuda",
                           "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-L/usr/local/cuda/lib64", "-lcudart",
                           "-Wl,-rpath,$ORIGIN"])
    os.replace(tmp, NATIVE)
    for o in objs:
        os.remove(o)
    with open(NATIVE + f".digest.{os.getpid()}", "w") as f:
        f.write(_native_digest())
    os.replace(NATIVE + f".digest.{os.getpid()}", NATIVE + ".digest")
    return NATIVE


def _stale() -> bool:
    """The library is current when the digest recorded beside it at build time matches the
    sources (file times are not used: they do not survive a copy of the tree)."""
    if not os.path.exists(LIB) or not os.path.exists(STAMP):
        return True
    with open(STAMP) as f:
        return f.read().strip() != _source_digest()


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile the library if it is missing or older than its sources."""
    if not force and not _stale():
        return LIB
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: cannot build libwkv_b200.so")
    objs = []
    bdir = os.path.join(PKG, "build")
    os.makedirs(bdir, exist_ok=True)
    procs = []
    for s in SOURCES:
        obj = os.path.join(bdir, s.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, s), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
            print(" ".join(cmd), flush=True)
        procs.append((s, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)))
        objs.append(obj)
    for s, p in procs:
        out = p.communicate()[0].decode()
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {s}:\n{out}")
        if verbose and out:
            print(out)
    # link beside the target and move into place: another process may be loading the library
    tmp = f"{LIB}.{os.getpid()}.tmp"
    subprocess.check_call([nvcc, "-shared", "-Xlinker", "-soname=libwkv_b200.so", "-o", tmp, *objs])
    os.replace(tmp, LIB)
    with open(STAMP + f".{os.getpid()}", "w") as f:
        f.write(_source_digest())
    os.replace(STAMP + f".{os.getpid()}", STAMP)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
    print(build_native(force="--force" in sys.argv))

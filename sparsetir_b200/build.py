"""Builds ``libsparsetir_b200.so`` in-tree with nvcc for sm_100a.

Usage: ``python -m sparsetir_b200.build [--force] [--verbose]``.
Objects go to ``build/`` at the repository root; the shared library is written next to this
file so that it travels with the source tree, and so is ``_pycall.so``, the Python extension
that packs torch tensors for it.
"""
from __future__ import annotations

import argparse
import concurrent.futures as cf
import os
import shutil
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG_DIR)
CSRC = os.path.join(PKG_DIR, "csrc")
INCLUDE = os.path.join(ROOT, "include")
OBJ_DIR = os.path.join(ROOT, "build", "obj")
LIB_PATH = os.path.join(PKG_DIR, "libsparsetir_b200.so")

PYCALL_PATH = os.path.join(PKG_DIR, "_pycall.so")

SOURCES = [
    "runtime.cc", "abi.cc", "format.cc", "validate.cu",
    "csrmm.cu", "csr_split.cu", "hyb_spmm.cu", "sddmm.cu", "bsrmm.cu", "bsrmm_tc.cu", "bsrmm_mma.cu", "rgms.cu", "rgms_tc.cu", "rgms_pairs.cu", "rgms_fused.cu", "rgms_wide.cu", "rgms_noalloc.cu", "rgms_ell3d.cu", "rgms_f16.cu", "sparse_conv.cu", "tcspmm.cu", "csr_misc.cu", "fusedmm.cu", "peer_scatter.cu",
]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "--extended-lambda", "-Xcompiler", "-fPIC,-fvisibility=hidden,-Wall",
    "-I", INCLUDE, "-I", CSRC,
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the library cannot be built")
    return exe


def _newest_header() -> float:
    newest = 0.0
    for d in (CSRC, INCLUDE):
        for f in os.listdir(d):
            if f.endswith((".h", ".cuh")):
                newest = max(newest, os.path.getmtime(os.path.join(d, f)))
    return newest


def _compile(src: str, force: bool, verbose: bool, hdr_mtime: float) -> str:
    obj = os.path.join(OBJ_DIR, src + ".o")
    path = os.path.join(CSRC, src)
    if (not force and os.path.exists(obj)
            and os.path.getmtime(obj) > max(os.path.getmtime(path), hdr_mtime)):
        return obj
    cmd = [_nvcc(), *NVCC_FLAGS, "-x", "cu", "-c", path, "-o", obj]
    if verbose:
        cmd.insert(1, "-Xptxas=-v")
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(f"$ {' '.join(cmd)}\n{res.stdout}{res.stderr}")
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src}")
    return obj


def build_pycall(force: bool = False, cuda: bool | None = None, out: str = PYCALL_PATH) -> str | None:
    """The extension module against this Python's and this torch's headers (g++).  Without torch there
    is nothing to pack and nothing is built; a torch without CUDA (``cuda=False``) has no streams to ask for."""
    try:
        import torch
    except ImportError:
        print("torch is not installed: building the library alone, without _pycall.so", file=sys.stderr)
        return None

    src = os.path.join(CSRC, "pycall.cc")
    torch_dir = os.path.dirname(os.path.abspath(torch.__file__))
    lib_dir = os.path.join(torch_dir, "lib")
    if cuda is None:
        cuda = torch.version.cuda is not None
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wall",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DSPTIR_TORCH_VERSION="{torch.__version__}"',
           f"-DSPTIR_TORCH_CUDA={int(cuda)}", "-I", INCLUDE,
           "-isystem", sysconfig.get_path("include"), "-isystem", os.path.join(torch_dir, "include"),
           "-isystem", os.path.join(torch_dir, "include", "torch", "csrc", "api", "include")]
    if cuda:
        cmd += ["-isystem", os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")]
    cmd += [src, "-o", out, "-L", lib_dir, f"-Wl,-rpath,{lib_dir}", "-ltorch_python", "-ltorch_cpu",
            *(["-lc10_cuda"] if cuda else []), "-lc10"]
    # the command names torch's version and folder and Python's headers: another one of them builds anew
    made_by = os.path.join(OBJ_DIR, "pycall.cmd") if out == PYCALL_PATH else out + ".cmd"
    key = "\n".join(cmd).replace(ROOT, "")  # wherever this tree lies
    newest = max(os.path.getmtime(src), os.path.getmtime(os.path.join(INCLUDE, "sparsetir_b200.h")))
    if not force and os.path.exists(out) and os.path.exists(made_by) and os.path.getmtime(out) > newest:
        with open(made_by) as f:
            if f.read() == key:
                return out
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(f"$ {' '.join(cmd)}\n{res.stdout}{res.stderr}")
        raise RuntimeError("g++ failed on pycall.cc")
    os.makedirs(os.path.dirname(made_by), exist_ok=True)
    with open(made_by, "w") as f:
        f.write(key)
    return out


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ_DIR, exist_ok=True)
    hdr = _newest_header()
    with cf.ThreadPoolExecutor(max_workers=min(8, len(SOURCES))) as pool:
        pycall = pool.submit(build_pycall, force)
        objs = list(pool.map(lambda s: _compile(s, force, verbose, hdr), SOURCES))
        pycall.result()
    if (force or not os.path.exists(LIB_PATH)
            or os.path.getmtime(LIB_PATH) < max(os.path.getmtime(o) for o in objs)):
        cmd = [_nvcc(), "-shared", "-o", LIB_PATH, *objs, "-gencode",
               "arch=compute_100a,code=sm_100a"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            sys.stderr.write(res.stdout + res.stderr)
            raise RuntimeError("link failed")
    return LIB_PATH


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))

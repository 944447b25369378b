"""Build libnova_b200.so in-tree with nvcc for sm_100a.

    python -m novaclone_b200.build          # incremental
    python -m novaclone_b200.build --force  # rebuild everything

Objects go to novaclone_b200/_build/, the shared library to
novaclone_b200/libnova_b200.so (found by novaclone_b200.nova at import).
"""
from __future__ import annotations

import argparse
import os
import re
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
BUILD = os.path.join(PKG, "_build")
LIB = os.path.join(PKG, "libnova_b200.so")
INCLUDE = os.path.join(ROOT, "include")
CUDA_HOME = os.environ.get("CUDA_HOME", "/usr/local/cuda")
NVCC = os.path.join(CUDA_HOME, "bin", "nvcc")

SOURCES = ["nova_stage.cu", "nova_stage_tma.cu", "nova_stage_mhd_tma.cu", "nova_proj_tma.cu", "nova_ops.cu", "nova_ex.cu", "nova_pois_i.cu", "nova_spec_row.cu", "nova_spec_col.cu",
    "nova_pois_dct.cu", "nova_fft2d.cu", "nova_adjoint.cu", "nova_adj_tma.cu", "nova_wc.cu", "nova_io.cu", "nova_im.cu", "nova_capi.cu"]
# sources compiled in parts (csrc/nova_parts.h): the number of parts, the last of them the dispatch
PARTS = {"nova_stage_tma.cu": 11, "nova_stage_mhd_tma.cu": 9, "nova_proj_tma.cu": 11, "nova_pois_i.cu": 7,
         "nova_spec_row.cu": 7, "nova_spec_col.cu": 7}
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-diag-suppress", "177", "-Xcompiler", "-fPIC", "-I" + INCLUDE, "-I" + CSRC]


def _newer(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _deps(path, seen=None):
    """path and the headers it includes from csrc/ and include/"""
    seen = set() if seen is None else seen
    if path in seen:
        return seen
    seen.add(path)
    for name in re.findall(r'^\s*#include "([^"]+)"', open(path).read(), re.M):
        for d in (CSRC, INCLUDE):
            if os.path.exists(os.path.join(d, name)):
                _deps(os.path.join(d, name), seen)
    return seen


def _jobs(force):
    """(object, nvcc command or None where it is up to date) of every source and part"""
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        deps = _deps(s)
        for p in range(PARTS.get(src, 1)):
            part = ["-DNOVA_PART=%d" % p] if src in PARTS else []
            o = os.path.join(BUILD, src[:-3] + ("_%d" % p if part else "") + ".o")
            yield o, [NVCC] + ARCH + FLAGS + part + ["-c", s, "-o", o] if force or _newer(o, deps) else None


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(BUILD, exist_ok=True)

    def compile(cmd):
        if verbose:
            print(" ".join(cmd))
        r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)
        if r.returncode != 0:
            sys.stderr.write(r.stdout.decode())
            raise RuntimeError("nvcc failed: " + " ".join(cmd))
    jobs = list(_jobs(force))
    with ThreadPoolExecutor(min(os.cpu_count() or 1, 16)) as pool:  # about 1 GB each
        list(pool.map(compile, [cmd for _, cmd in jobs if cmd]))
    objs = [o for o, _ in jobs]
    if force or _newer(LIB, objs):
        cmd = [NVCC] + ARCH + ["-shared", "-o", LIB] + objs + [
            "-L" + os.path.join(CUDA_HOME, "lib64"), "-lcufft",
            "-Xlinker", "-rpath," + os.path.join(CUDA_HOME, "lib64"),
            "-Xlinker", "-z", "-Xlinker", "defs"]  # a part that is missing fails here
        if verbose:
            print(" ".join(cmd))
        subprocess.run(cmd, check=True)
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=True))

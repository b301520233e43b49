"""Build liblitedsa_b200.so (all CUDA kernels + the C ABI) in-tree with nvcc for sm_100a.

    python -m litetopk_b200.build [--force] [--verbose]

The library lands in litetopk_b200/_C/ (git-ignored, but shipped with the source tree to
the GPU machine).  Only nvcc and the CUDA runtime are needed: no CUTLASS, no Python
headers, no torch headers.  Beside it, litedsa_host-*.so, the short way from Python to the library's
calls (csrc/host_binding.cpp), needs both and is one interpreter's and one torch's; where it cannot be built
the package goes by ctypes alone.
"""
from __future__ import annotations

import argparse
import os
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OUT_DIR = PKG / "_C"
LIB = OUT_DIR / "liblitedsa_b200.so"
HOST_SRC = CSRC / "host_binding.cpp"
SOURCES = ["abi.cu", "union_qm.cu", "attn_fp8.cu", "prep.cu", "noalloc.cu", "attn_dsv4.cu", "attn_bf16.cu", "peak_probe.cu", "index_topk.cu",
           "prefill.cu"]


def _nvcc() -> str:
    home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    return str(Path(home) / "bin" / "nvcc")


def sources():
    return [CSRC / s for s in SOURCES]


def is_stale() -> bool:
    if not LIB.exists():
        return True
    t = LIB.stat().st_mtime
    deps = list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + \
        [PKG.parent / "include" / "litedsa_b200.h", Path(__file__)]
    return any(d.stat().st_mtime > t for d in deps)


def build_host(verbose: bool = False) -> None:
    """The module of host_binding.cpp for this interpreter and torch, linked against the library beside it, unless it is there;
    modules of an earlier library, whoever's they are, leave."""
    newest = max(HOST_SRC.stat().st_mtime, LIB.stat().st_mtime)
    for f in OUT_DIR.glob("litedsa_host*.so"):
        if f.stat().st_mtime < newest:
            f.unlink()
    try:
        import sysconfig
        import torch
        from torch.utils import cpp_extension as ext
        from ._lib import host_path
        path = OUT_DIR / host_path().name
        if path.exists():
            return
        includes = [sysconfig.get_paths()["include"], *ext.include_paths(), str(Path(_nvcc()).parents[1] / "include")]
        tmp = path.with_suffix(".so.tmp")
        cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-I{d}" for d in includes), str(HOST_SRC), "-o", str(tmp),
               *(f"-L{d}" for d in ext.library_paths()), "-ltorch", "-ltorch_cpu", "-ltorch_python", "-lc10", "-lc10_cuda",
               f"-L{OUT_DIR}", f"-l:{LIB.name}", "-Wl,-rpath,$ORIGIN"]
        if verbose:
            print(" ".join(cmd), flush=True)
        p = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if p.returncode != 0:
            raise RuntimeError(p.stdout[-2000:])
        os.replace(tmp, path)
    except Exception as e:      # no Python or torch headers, no g++: the package goes by ctypes
        sys.stderr.write(f"the module of {HOST_SRC.name} was not built: {e}\n")


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and not is_stale():
        build_host(verbose)
        return LIB
    OUT_DIR.mkdir(exist_ok=True)
    objs = []
    procs = []
    for src in sources():
        obj = OUT_DIR / (src.stem + ".o")
        cmd = [_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3",
               "-std=c++17", "-use_fast_math", "--compiler-options=-fPIC", "-c", str(src),
               "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
            print(" ".join(cmd), flush=True)
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(out)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src.name}")
    tmp = LIB.with_suffix(".so.tmp")
    cmd = [_nvcc(), "-shared", "-o", str(tmp)] + [str(o) for o in objs] + ["-lcudart"]
    subprocess.check_call(cmd)
    os.replace(tmp, LIB)
    build_host(verbose)
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))

"""In-tree build of libevoattn.so (sm_100a only).

    python megakernel-exploration_b200/build.py [--force] [--verbose]

Each csrc/*.cu is compiled with nvcc for compute_100a/sm_100a and the objects
are linked into megakernel-exploration_b200/libevoattn.so next to this file.
nvcc cross-compiles, so no GPU is needed to build.  The library links the CUDA
runtime statically and resolves the driver's tensor-map encoder at run time,
so it also loads on a machine without a driver (compute calls then fail with
EVO_ERR_NO_DRIVER / EVO_ERR_CUDA).  csrc/evo_torch.cpp becomes _evo_torch.so, the
operator's native host path.
"""
from __future__ import annotations

import argparse
import concurrent.futures as cf
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ_DIR = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libevoattn.so")
EXT = os.path.join(HERE, "_evo_torch.so")       # the operator's native host path (needs torch's headers)
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-Xptxas", "-v",
    "--expt-relaxed-constexpr",
]


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _deps_mtime():
    m = 0.0
    for d in (CSRC, INCLUDE):
        for f in os.listdir(d):
            if f.endswith((".cu", ".cuh", ".h", ".cpp")):
                m = max(m, os.path.getmtime(os.path.join(d, f)))
    return max(m, os.path.getmtime(__file__))


def _compile(src: str, verbose: bool) -> str:
    obj = os.path.join(OBJ_DIR, src[:-3] + ".o")
    cmd = ["nvcc", *NVCC_FLAGS, "-I", INCLUDE, "-c", os.path.join(CSRC, src), "-o", obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
    log = os.path.join(OBJ_DIR, src[:-3] + ".ptxas.log")
    with open(log, "w") as f:
        f.write(r.stderr)
    if verbose:
        sys.stderr.write(r.stderr)
    return obj


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile (if stale) and return the path of libevoattn.so."""
    if not force and all(os.path.exists(f) and os.path.getmtime(f) >= _deps_mtime() for f in (LIB, EXT)):
        return LIB
    os.makedirs(OBJ_DIR, exist_ok=True)
    srcs = _sources()
    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(lambda s: _compile(s, verbose), srcs))
    cmd = ["nvcc", "-shared", "-o", LIB, *objs, "-cudart", "static"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    _build_ext()
    return LIB


def _build_ext() -> None:
    """_evo_torch.so: csrc/evo_torch.cpp against torch and libevoattn.so (found next to it at run time)."""
    import sysconfig
    import torch
    from torch.utils import cpp_extension as ce
    src = os.path.join(CSRC, "evo_torch.cpp")
    inc = [a for d in (*ce.include_paths(device_type="cuda"), sysconfig.get_paths()["include"]) for a in ("-isystem", d)]
    lib = [a for d in ce.library_paths(device_type="cuda") for a in (f"-L{d}", f"-Wl,-rpath,{d}")]
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wall", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-DTORCH_EXTENSION_NAME=_evo_torch", "-DTORCH_API_INCLUDE_EXTENSION_H", *inc, src, "-o", EXT, "-Wl,-rpath,$ORIGIN",
           f"-L{HERE}", "-l:libevoattn.so", *lib, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for {src}:\n{r.stderr[-8000:]}")


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))

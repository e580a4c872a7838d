"""Builds ``vortex_b200/lib/libvortex_b200.so`` from ``vortex_b200/csrc/*.cu`` with nvcc for sm_100a, and the host
module ``vortex_b200/lib/_vtx_host.so`` from ``csrc/host.cpp`` with g++ against torch's and Python's headers.

    python -m vortex_b200.build [--force] [--verbose]
    python vortex_b200/build.py          # the same where torch is not installed: the library (C ABI) alone

nvcc cross-compiles without a GPU.  Objects are rebuilt only when their source (or a header)
changed.  The library is kept in-tree so that it travels with the checkout.
"""
from __future__ import annotations

import argparse
import concurrent.futures as cf
import hashlib
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIBDIR = os.path.join(PKG, "lib")
OBJDIR = os.path.join(LIBDIR, "obj")
LIB = os.path.join(LIBDIR, "libvortex_b200.so")
HOST_SRC, HOST_LIB = os.path.join(CSRC, "host.cpp"), os.path.join(LIBDIR, "_vtx_host.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-Xptxas", "-v",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC=/path/to/nvcc)")


def _digest(paths) -> str:
    h = hashlib.sha256(" ".join(NVCC_FLAGS).encode())
    for p in sorted(paths):
        with open(p, "rb") as f:
            h.update(p.encode() + b"\0" + f.read())
    return h.hexdigest()


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def headers():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs.append(os.path.join(os.path.dirname(PKG), "include", "vortex_b200.h"))
    return sorted(hs)


def _compile(src: str, force: bool, verbose: bool) -> tuple[str, bool, str]:
    obj = os.path.join(OBJDIR, os.path.basename(src)[:-3] + ".o")
    stamp = obj + ".sha"
    want = _digest([src] + headers())
    if not force and os.path.exists(obj) and os.path.exists(stamp) and open(stamp).read() == want:
        return obj, False, ""
    cmd = [_nvcc()] + NVCC_FLAGS + ["-c", src, "-o", obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
    with open(stamp, "w") as f:
        f.write(want)
    return obj, True, r.stderr if verbose else ""


def _build_host(force: bool) -> None:
    import sysconfig

    try:
        import torch
    except ImportError:          # the module serves the Python wrappers, which need torch; the C ABI does not
        print("torch not found: host module not built", file=sys.stderr)
        return
    from torch.utils import cpp_extension as ext

    stamp = os.path.join(OBJDIR, "host.sha")
    want = _digest([HOST_SRC, os.path.join(os.path.dirname(PKG), "include", "vortex_b200.h")]) + torch.__version__ + sysconfig.get_python_version()
    if not force and os.path.exists(HOST_LIB) and os.path.exists(stamp) and open(stamp).read() == want:
        return
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    libdir = os.path.join(os.path.dirname(torch.__file__), "lib")
    inc = [*ext.include_paths(), os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wall", "-DTORCH_API_INCLUDE_EXTENSION_H",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-isystem{d}" for d in inc), HOST_SRC,
           "-o", HOST_LIB, f"-L{libdir}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for {HOST_SRC}:\n{r.stdout}\n{r.stderr}")
    with open(stamp, "w") as f:
        f.write(want)


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJDIR, exist_ok=True)
    srcs = sources()
    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs)) + 1) as ex:
        host = ex.submit(_build_host, force)
        results = list(ex.map(lambda s: _compile(s, force, verbose), srcs))
    objs = [o for o, _, _ in results]
    if verbose:
        for _, _, log in results:
            if log:
                print(log, file=sys.stderr)
    # (an object newer than the library: an earlier build ended between the two)
    if any(changed for _, changed, _ in results) or not os.path.exists(LIB) or \
            max(map(os.path.getmtime, objs)) > os.path.getmtime(LIB):
        cmd = [_nvcc(), "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    host.result()                # (raises what the host module's build raised, the library being linked)
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))

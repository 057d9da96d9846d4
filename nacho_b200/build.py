"""Builds ``libnacho_b200.so`` (CUDA kernels + C ABI) for sm_100a with nvcc and ``_native.so`` (the
Python operators over it) with g++, in-tree.

Run as ``python -m nacho_b200.build``. Objects are cached under ``nacho_b200/csrc/build/``
and rebuilt when a source or header is newer.
"""
from __future__ import annotations

import concurrent.futures as cf
import glob
import os
import re
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
OBJ_DIR = os.path.join(CSRC, "build")
LIB = os.path.join(HERE, "libnacho_b200.so")
NATIVE = os.path.join(HERE, "_native.so")
NATIVE_FOR = os.path.join(OBJ_DIR, "native.txt")  # the interpreter and the torch that it was built for

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "--fmad=false",  # bit-exact parity: a * b followed by + must not contract
    "-Xcompiler", "-fPIC,-O3",
    "-I", os.path.join(ROOT, "include"), "-I", CSRC,
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the nacho_b200 library cannot be built")


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _read(path: str) -> str | None:
    if not os.path.exists(path):
        return None
    with open(path) as f:
        return f.read()


def _report(obj: str) -> str:
    return obj[:-2] + ".ptxas.txt"


def spills(name: str) -> dict[str, tuple[int, int]]:
    """Bytes of spill stores and loads of every device function of ``csrc/<name>.cu``, by mangled name, as ptxas reported them."""
    text = _read(_report(os.path.join(OBJ_DIR, name + ".o"))) or ""
    found = re.findall(r"Function properties for (\S+)\n\s*\d+ bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads", text)
    return {f: (int(stores), int(loads)) for f, stores, loads in found}


def build(verbose: bool = False, ptxas_info: bool = False) -> str:
    nvcc = _nvcc()
    os.makedirs(OBJ_DIR, exist_ok=True)
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    headers = sorted(glob.glob(os.path.join(CSRC, "*.cuh"))) + sorted(glob.glob(os.path.join(ROOT, "include", "*.h")))
    headers.append(os.path.abspath(__file__))
    jobs = []
    objs = []
    for src in sources:
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if _stale(obj, [src] + headers) or not os.path.exists(_report(obj)):
            jobs.append([nvcc] + NVCC_FLAGS + ["-Xptxas", "-v", "-c", src, "-o", obj])

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        with open(_report(cmd[-1]), "w") as f:
            f.write(r.stderr)
        return cmd, r

    with cf.ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for cmd, r in ex.map(run, jobs):
            if verbose or ptxas_info or r.returncode != 0:
                sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + (r.stderr if ptxas_info or r.returncode != 0 else ""))
            if r.returncode != 0:
                raise RuntimeError(f"nvcc failed for {cmd[-3]}")
    if jobs or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", LIB, "-Xlinker", "-soname=libnacho_b200.so"] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link of libnacho_b200.so failed")
    build_native(nvcc, verbose)
    return LIB


def build_native(nvcc: str, verbose: bool = False) -> str | None:
    """``_native.so`` against the torch of this interpreter; it finds ``libnacho_b200.so`` beside itself. Rebuilt when a source
    is newer or it was built for another interpreter or torch. The C library needs neither: without a torch this says so
    and builds nothing."""
    try:
        import torch
    except ImportError:
        sys.stderr.write("torch is not installed: nacho_b200/_native.so, the Python operators, is not built\n")
        return None
    src = os.path.join(CSRC, "native.cpp")
    built_for = f"python {sys.version}\ntorch {torch.__version__} {torch.version.git_version}\n"
    if not _stale(NATIVE, [src, os.path.join(ROOT, "include", "nacho_b200.h"), os.path.abspath(__file__)]) and _read(NATIVE_FOR) == built_for:
        return NATIVE
    torch_dir = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc)))
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for inc in (os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"),
                os.path.join(cuda, "include"), sysconfig.get_paths()["include"]):
        cmd += ["-isystem", inc]
    cmd += ["-I", os.path.join(ROOT, "include"), src, "-o", NATIVE, "-L", os.path.join(torch_dir, "lib"), "-L", HERE, "-lnacho_b200",
            "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode != 0:
        sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError("build of _native.so failed")
    with open(NATIVE_FOR, "w") as f:
        f.write(built_for)
    return NATIVE


if __name__ == "__main__":
    path = build(verbose="-v" in sys.argv, ptxas_info="--ptxas" in sys.argv)
    print(path)

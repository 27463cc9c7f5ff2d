"""Build in-tree: liblampa_b200.so (the C-ABI CUDA library, nvcc for sm_100a) and _host.so (the native host path of the
Python entry points, g++ against torch's headers and the library)."""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
SO = os.path.join(HERE, "liblampa_b200.so")
HOST_SO = os.path.join(HERE, "_host.so")
HOST_SOURCES = ["host.cpp", "host_lsh.inc", "host_model.inc", "host_hept.inc"]
SOURCES = ["lsh.cu", "geo.cu", "layer.cu", "model.cu", "bucket_attn.cu", "gdn_prep.cu", "gdn_prep_umma.cu", "gdn_scan.cu", "gdn_scan_umma.cu", "gdn_state.cu", "gdn_api.cu", "profile.cu"]
HEADERS = ["common.cuh", "gdn.cuh", "gdn_inv.cuh", "gdn_load.cuh", "umma.cuh", "tmap.cuh", "act.cuh", "split3.cuh", "profile.cuh", os.path.join("..", "..", "include", "lampa_b200.h")]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _stale() -> bool:
    if not os.path.exists(SO):
        return True
    t = os.path.getmtime(SO)
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS]
    return any(os.path.getmtime(os.path.normpath(d)) > t for d in deps)


def _build_host(verbose: bool) -> None:
    import sysconfig
    import torch
    t = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.sep in _nvcc() else "/usr/local/cuda"
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", f"-I{t}/include",
           f"-I{t}/include/torch/csrc/api/include", f"-I{sysconfig.get_paths()['include']}", f"-I{cuda}/include",
           os.path.join(CSRC, "host.cpp"), "-o", HOST_SO, f"-L{t}/lib", "-lc10", "-lc10_cuda", "-ltorch_cpu",
           "-ltorch_cuda", "-ltorch_python", f"-L{HERE}", "-l:liblampa_b200.so", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError("g++ failed on host.cpp")


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu for sm_100a and link the shared library next to this file, then the host module."""
    built = force or _stale()
    if built:
        _build_library(verbose)
    host = [os.path.join(CSRC, f) for f in HOST_SOURCES] + [os.path.join(HERE, "..", "include", "lampa_b200.h")]
    if built or not os.path.exists(HOST_SO) or any(os.path.getmtime(f) > os.path.getmtime(HOST_SO) for f in host):
        _build_host(verbose)
    return SO


def _build_library(verbose: bool) -> None:
    nvcc = _nvcc()
    extra = os.environ.get("LAMPA_NVCC_EXTRA", "").split()   # extra nvcc flags
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)

    def compile_one(src: str) -> str:
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        cmd = [nvcc] + NVCC_FLAGS + extra + (["-Xptxas", "-v"] if verbose else []) + ["-c", os.path.join(CSRC, src), "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}")
        return obj

    with ThreadPoolExecutor(max_workers=6) as ex:
        objs = list(ex.map(compile_one, SOURCES))
    r = subprocess.run([nvcc, "-shared", "-o", SO] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"],
                       capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("link failed")


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))

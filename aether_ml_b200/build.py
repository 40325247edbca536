"""Builds libaether_b200.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a.

    python -m aether_ml_b200.build            # or: from aether_ml_b200.build import build_library
"""
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_PATH = os.path.join(HERE, "libaether_b200.so")
DIGEST_PATH = LIB_PATH + ".digest"
HOST_PATH = os.path.join(HERE, "_host.so")          # native host path: a CPython module against torch's C++ interface
HOST_DIGEST_PATH = HOST_PATH + ".digest"
HOST_SOURCE = os.path.join(CSRC, "host.cpp")
HEADER = os.path.join(HERE, "..", "include", "aether_b200.h")
HOST_FLAGS = ["-O2", "-std=c++17", "-shared", "-fPIC"]
SOURCES = ["api.cu", "conv_tc.cu", "conv_halo.cu", "conv_halo_dw.cu", "conv_dw_rows.cu", "conv_generic.cu", "conv_dx_few.cu", "conv_simt.cu", "conv_split.cu", "conv_smallc.cu", "conv_first_tc.cu", "conv_first_fp32.cu", "layers.cu",
           "block_fused.cu", "bn_small.cu"]
# tcgen05 / TMA PTX only assembles for the arch-specific target, hence compute_100a + sm_100a.
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC"]


def _nvcc():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; cannot build libaether_b200.so")
    return nvcc


def _digest(paths, seed):
    """sha256 over files and what else the built file is a function of."""
    import hashlib
    h = hashlib.sha256(seed.encode())
    for d in paths:
        h.update(os.path.basename(d).encode())
        with open(d, "rb") as fh:
            h.update(fh.read())
    return h.hexdigest()


def _source_digest():
    cuda = sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))
    return _digest(cuda + [HEADER], " ".join(NVCC_FLAGS))


def _host_digest():
    import torch
    return _digest([HOST_SOURCE, HEADER], " ".join(HOST_FLAGS) + torch.__version__ + sys.version)


def _current(path, digest_path, digest):
    """False when a built file is missing or was built from other sources.  The check compares a digest of the
    sources with the one recorded beside the .so at build time, so it does not depend on file times (a copied
    tree keeps its built files)."""
    if not os.path.exists(path) or not os.path.exists(digest_path):
        return False
    with open(digest_path) as fh:
        return fh.read().strip() == digest


def _stale():
    return not (_current(LIB_PATH, DIGEST_PATH, _source_digest()) and _current(HOST_PATH, HOST_DIGEST_PATH, _host_digest()))


def build_host(force=False):
    """Compile the native host module if it is missing or older than its sources.  Returns its path."""
    digest = _host_digest()
    if not force and _current(HOST_PATH, HOST_DIGEST_PATH, digest):
        return HOST_PATH
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME") or os.path.dirname(os.path.dirname(_nvcc()))
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    cmd = ([os.environ.get("CXX", "g++")] + HOST_FLAGS + ["-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI]
           + ["-I" + p for p in include] + [HOST_SOURCE, "-o", HOST_PATH, "-L" + os.path.join(root, "lib")]
           + ["-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-ldl"])
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("%s failed for host.cpp:\n%s\n%s" % (cmd[0], r.stdout, r.stderr))
    with open(HOST_DIGEST_PATH, "w") as fh:
        fh.write(digest + "\n")
    return HOST_PATH


def build_library(force=False, verbose=False):
    """Compile the library and the native host module if they are missing or older than their sources.  Returns the
    library's path."""
    build_host(force)
    if not force and _current(LIB_PATH, DIGEST_PATH, _source_digest()):
        return LIB_PATH
    nvcc = _nvcc()
    build_dir = os.path.join(HERE, "build")
    os.makedirs(build_dir, exist_ok=True)

    def compile_one(src):
        obj = os.path.join(build_dir, src.replace(".cu", ".o"))
        cmd = [nvcc, "-c", os.path.join(CSRC, src), "-o", obj] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else [])
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed for %s:\n%s\n%s" % (src, r.stdout, r.stderr))
        if verbose:
            print(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
        objs = list(pool.map(compile_one, SOURCES))
    cmd = [nvcc, "-shared", "-o", LIB_PATH] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n%s\n%s" % (r.stdout, r.stderr))
    with open(DIGEST_PATH, "w") as fh:
        fh.write(_source_digest() + "\n")
    return LIB_PATH


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))

"""Build recipe of libwhir_gb300.so (sm_103a kernels + C++ host + C ABI).

Compiles every translation unit in parallel with nvcc for
``-gencode arch=compute_103a,code=sm_103a`` and links an in-tree shared
library at whir_gb300/_lib/libwhir_gb300.so.  Objects go to
whir_gb300/_build/.  Rebuilds only what changed.
"""

import concurrent.futures as cf
import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
BUILD = os.path.join(HERE, "_build")
LIBDIR = os.path.join(HERE, "_lib")
LIB = os.path.join(LIBDIR, "libwhir_gb300.so")

CU_SOURCES = ["ntt.cu", "merkle.cu", "merkle_tensor.cu", "sumcheck.cu", "noalloc.cu"]
CPP_SOURCES = ["poseidon2_host.cpp", "p2_matrix.cpp", "transcript.cpp", "svo_host.cpp", "prover.cpp", "batch_prover.cpp", "batch.cpp", "verifier.cpp", "verify_batch.cpp", "tune.cpp",
               "capi.cpp"]
HOST_SOURCES = ["poseidon2_host.cpp"]  # vector types: not through nvcc's front end
GENCODE = ["-gencode", "arch=compute_103a,code=sm_103a"]


def nvcc():
    path = shutil.which("nvcc")
    if path:
        return path
    cand = "/usr/local/cuda/bin/nvcc"
    if os.path.exists(cand):
        return cand
    raise RuntimeError("nvcc not found")


def _headers():
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))] + [
        os.path.join(INCLUDE, "whir_gb300.h")]


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _compile(src, verbose):
    path = os.path.join(CSRC, src)
    obj = os.path.join(BUILD, src + ".o")
    if not _stale(obj, [path] + _headers()):
        return obj
    cmd = [nvcc(), *GENCODE, "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC",
           "-Xcompiler", "-fvisibility=hidden", "-I", CSRC, "-I", INCLUDE, "-c", path, "-o", obj]
    if src.endswith(".cpp") and src not in HOST_SOURCES:
        cmd[1:1] = ["-x", "cu"]
    if verbose:
        cmd.append("-Xptxas=-v")
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
    if verbose and r.stderr:
        print(r.stderr)
    return obj


def build(verbose=False, force=False):
    """Compile and link; returns the library path."""
    os.makedirs(BUILD, exist_ok=True)
    os.makedirs(LIBDIR, exist_ok=True)
    if force:
        for f in os.listdir(BUILD):
            os.remove(os.path.join(BUILD, f))
    srcs = CU_SOURCES + CPP_SOURCES
    with cf.ThreadPoolExecutor(max_workers=len(srcs)) as ex:
        objs = list(ex.map(lambda s: _compile(s, verbose), srcs))
    if _stale(LIB, objs):
        cmd = [nvcc(), *GENCODE, "-shared", "-o", LIB, *objs, "-lcudart_static", "-lrt",
               "-lpthread", "-ldl"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return LIB


if __name__ == "__main__":
    import sys
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))

"""Builds ``libcphnsw_b200.so`` (the C-ABI library declared in ``include/cphnsw_b200.h``) in-tree.

    python sparse-text-kmeans_b200/build.py [--force] [--verbose]

nvcc cross-compiles for sm_100a without a GPU.  ``--fmad=false`` keeps every fp32 add of the
transform and of the score accumulation a separate IEEE operation (the dot products of the
rerank call fmaf explicitly).
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libcphnsw_b200.so")
SOURCES = ["api.cu", "device_memory.cu", "encode.cu", "distance.cu", "knn_sliced.cu", "knn_mma.cu", "search.cu", "search_walk.cu", "multiprobe.cu", "diagnostics.cu", "exact.cu", "exact_mma.cu", "rank_prune.cu", "sharded.cu", "exact_edges.cu"]
HEADERS = [os.path.join(CSRC, "common.cuh"), os.path.join(CSRC, "knn_common.cuh"), os.path.join(CSRC, "mma_common.cuh"), os.path.join(CSRC, "search_common.cuh"), os.path.join(HERE, "..", "include", "cphnsw_b200.h")]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "--fmad=false", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    nvcc = _nvcc()
    objs = []
    procs = []
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        o = os.path.join(HERE, "build", src.replace(".cu", ".o"))
        objs.append(o)
        if force or _stale(o, [s] + HEADERS):
            cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write("== %s ==\n%s\n" % (src, out))
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    if force or procs or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB] + objs + ["-ldl"]
        subprocess.check_call(cmd)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))

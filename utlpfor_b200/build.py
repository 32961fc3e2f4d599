"""Build the CUDA library in-tree: utlpfor_b200/libutlpfor_b200.so (sm_100a).

    python -m utlpfor_b200.build          # or build() from Python
"""
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libutlpfor_b200.so")
SOURCES = ["utl_kernels.cu", "utl_pack.cu", "utl_get.cu", "utl_capi.cu", "utl_noalloc.cu", "utl_index.cu"]
HEADERS = ["utl_device.cuh", "utl_launch.h", "utl_quad.cuh", "utl_lane.cuh", "utl_pieces.h", "utl_unpack.cuh", "utl_pair.cuh",
           "utl_unlane.cuh", "utl_get.cuh",
           "utl_qpack.cuh", "utl_streams.cuh"]
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def nvcc_path():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _stale():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS]
    deps.append(os.path.join(os.path.dirname(HERE), "include", "utlpfor.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    if not force and not _stale():
        return LIB
    cmd = [nvcc_path(), *ARCH, "-lineinfo", "-O3", "-std=c++17", "--threads", "0", "-shared", "-Xcompiler", "-fPIC",
           "-Xcompiler", "-fvisibility=hidden", "-o", LIB + ".tmp"]
    cmd += [os.path.join(CSRC, f) for f in SOURCES]
    if verbose:
        cmd.insert(1, "-Xptxas=-v")
        print(" ".join(cmd))
    subprocess.check_call(cmd)
    os.replace(LIB + ".tmp", LIB)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(LIB)

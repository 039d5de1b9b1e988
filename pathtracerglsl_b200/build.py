"""Build recipe of the CUDA library ``pathtracerglsl_b200/libptx_rt.so`` (sm_100a).

nvcc cross-compiles without a GPU; the shared object is built in-tree so it travels
with the working tree.  ``-fmad=false`` keeps every product and sum rounded as written
(binary32 in the operation order of the reference's shader math).
"""
import glob
import os
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libptx_rt.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-lineinfo", "-std=c++17", "-fmad=false", "-Xcompiler", "-fPIC,-O3,-ffp-contract=off", "-split-compile=4"]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "**", "*.cu"), recursive=True) +
                  glob.glob(os.path.join(CSRC, "**", "*.cuh"), recursive=True) +
                  glob.glob(os.path.join(CSRC, "**", "*.cpp"), recursive=True) +
                  glob.glob(os.path.join(CSRC, "**", "*.h"), recursive=True) +
                  [os.path.join(ROOT, "include", "ptx_rt.h")])


def build(force=False, verbose=False):
    newest = max(os.path.getmtime(p) for p in sources())
    if not force and os.path.exists(LIB) and os.path.getmtime(LIB) >= newest:
        return LIB
    units = sorted(glob.glob(os.path.join(CSRC, "*.cu"))) + sorted(glob.glob(os.path.join(CSRC, "host", "*.cpp")))
    objs = []
    procs = []
    with tempfile.TemporaryDirectory() as tmp:   # the units compile side by side
        for u in units:
            objs.append(os.path.join(tmp, os.path.basename(u) + ".o"))
            cmd = [NVCC, *ARCH, *FLAGS, "-I", os.path.join(ROOT, "include"), "-I", os.path.join(CSRC, "device"), "-c", u, "-o", objs[-1]]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            procs.append(subprocess.Popen(cmd, stdout=subprocess.DEVNULL, stderr=subprocess.PIPE, text=True))
        errors = [p.communicate()[1] for p in procs]
        for p, err in zip(procs, errors):
            if p.returncode != 0:
                raise RuntimeError("nvcc failed:\n" + err[-4000:])
        r = subprocess.run([NVCC, *ARCH, "-shared", *objs, "-o", LIB + ".tmp"], capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc link failed:\n" + r.stderr[-4000:])
    os.replace(LIB + ".tmp", LIB)
    return LIB


if __name__ == "__main__":
    print(build(force=True, verbose=True))

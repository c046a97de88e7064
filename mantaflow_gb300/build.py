"""Build libmantagpu.so (sm_103a) in-tree with nvcc.

The library is a plain C-ABI shared object (include/mantagpu.h); Python
reaches it through ctypes.  -fmad=false keeps a*b+c uncontracted so the
kernels repeat the reference's float arithmetic exactly; the few places that
emulate the reference's double-rounded expressions call fmaf explicitly.  The
host compiler gets -ffp-contract=off for the same reason: the host-side set-up
arithmetic (the wavelet noise tile, shape axes, force factors) must not be
contracted into fused multiply-adds, which aarch64 gcc does by default.
"""
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libmantagpu.so")
SOURCES = ["runtime.cu", "advect.cu", "forces.cu", "pressure.cu", "cgcluster.cu", "mic.cu", "micwave.cu", "micflow.cu", "miccluster.cu", "multigrid.cu", "refine.cu", "batch.cu", "gridio.cu", "noise.cu", "particles.cu"]
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-fmad=false", "-Xcompiler", "-fPIC,-O2,-ffp-contract=off", "--expt-relaxed-constexpr"]


def nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: the CUDA toolkit is required to build libmantagpu")
    return exe


def _stale(out, deps):
    if not os.path.exists(out):
        return True
    t = os.path.getmtime(out)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    os.makedirs(BUILD, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    headers.append(os.path.join(os.path.dirname(HERE), "include", "mantagpu.h"))
    objs = []
    jobs = []
    for src in SOURCES:
        sp = os.path.join(CSRC, src)
        obj = os.path.join(BUILD, src + ".o")
        objs.append(obj)
        if force or _stale(obj, [sp] + headers):
            jobs.append([nvcc()] + ARCH + FLAGS + ["-c", sp, "-o", obj])

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed:\n%s\n%s" % (" ".join(cmd), r.stderr))
        if verbose and r.stderr:
            sys.stderr.write(r.stderr)

    with ThreadPoolExecutor(max_workers=len(SOURCES)) as ex:
        list(ex.map(run, jobs))
    if force or jobs or _stale(LIB, objs):
        run([nvcc()] + ARCH + ["-shared", "-o", LIB] + objs + ["-lcudart_static", "-lrt", "-lpthread", "-ldl"])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))

"""Build libkerrsplat_b200.so in-tree with nvcc for sm_100a (B200)."""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libkerrsplat_b200.so")
SOURCES = ["ks_lib.cu", "ks_forward.cu", "ks_reverse.cu"]
HEADERS = ["ks_elliptic.cuh", "ks_plan.cuh", "ks_march.cuh", "ks_dual.cuh", "ks_transfer.cuh", "ks_mixed.cuh", "ks_adjoint.cuh", "ks_spacetime.cuh", "ks_dft.cuh", "ks_context.cuh", "ks_transport.cuh", "ks_gradient.cuh", "ks_reverse.cuh", "ks_march_block.cuh"]


def nvcc_flags():
    """FP32 division and square root take the hardware approximations (-prec-div=false,
    -prec-sqrt=false: a few ulp, inside the mixed path's 1e-4 budget; the coefficient fits divide
    often and the IEEE sequences cost them a quarter of their time). FP64 arithmetic is unaffected,
    denormals are kept."""
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    return [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
            "--use_fast_math" if os.environ.get("KS_FAST_MATH") else "-Xptxas=-O3",
            "-prec-div=false", "-prec-sqrt=false", "-Xcompiler", "-fPIC"]


def _newest(paths):
    return max(os.path.getmtime(p) for p in paths)


def _dependencies():
    return [os.path.join(CSRC, h) for h in HEADERS] + [os.path.join(HERE, "..", "include", "kerrsplat_b200.h")]


def stale():
    return not os.path.exists(LIB) or _newest(_dependencies() + [os.path.join(CSRC, s) for s in SOURCES]) > os.path.getmtime(LIB)


def build(force=False, verbose=True):
    """Compile the CUDA library if a source is newer than the .so (or `force`): one object per source,
    side by side, then the link."""
    if not force and not stale():
        return LIB
    flags, objects, running = nvcc_flags(), [], []
    for s in SOURCES:
        src, obj = os.path.join(CSRC, s), os.path.join(CSRC, s.replace(".cu", ".o"))
        objects.append(obj)
        if not force and os.path.exists(obj) and os.path.getmtime(obj) > _newest(_dependencies() + [src]):
            continue
        cmd = flags + ["-c", src, "-o", obj]
        if verbose:
            print(" ".join(cmd), file=sys.stderr)
        running.append((cmd, subprocess.Popen(cmd)))
    for cmd, p in running:
        if p.wait() != 0:
            for obj in objects:   # no half-built object is left to be linked
                if obj == cmd[-1] and os.path.exists(obj):
                    os.remove(obj)
            raise subprocess.CalledProcessError(p.returncode, cmd)
    cmd = flags + ["-shared", "-o", LIB] + objects
    if verbose:
        print(" ".join(cmd), file=sys.stderr)
    subprocess.run(cmd, check=True)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv)

"""Build libkerrsplat_b200.so in-tree with nvcc for sm_100a (B200)."""
import fcntl
import hashlib
import os
import subprocess
import sys
import time

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libkerrsplat_b200.so")
OBJECTS = os.path.join(HERE, "_build")
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


def _tag():
    """The compiler and its flags: objects of other flags lie in other folders."""
    return hashlib.sha256("\0".join(nvcc_flags()).encode()).hexdigest()[:16]


def _built_with():
    """The tag of the library that is there (None: not known)."""
    stamp = os.path.join(OBJECTS, "tag")
    return open(stamp).read() if os.path.exists(stamp) else None


def stale():
    return not os.path.exists(LIB) or _built_with() not in (None, _tag()) or \
        _newest(_dependencies() + [os.path.join(CSRC, s) for s in SOURCES]) > os.path.getmtime(LIB)


def _put(tmp, path, when):
    """A finished file into its place, as old as the start of its build: a source edited since then is newer."""
    os.utime(tmp, (when, when))
    os.replace(tmp, path)


def build(force=False, verbose=True):
    """Compile the CUDA library if a source is newer than the .so, if it was built with other flags, or with `force`: one
    object per source, side by side, then the link. One process builds at a time, the others wait for it; nothing
    half-written lies under a name that is read."""
    if not force and not stale():
        return LIB
    folder = os.path.join(OBJECTS, _tag())
    os.makedirs(folder, exist_ok=True)
    with open(os.path.join(OBJECTS, "lock"), "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        if not force and not stale():
            return LIB
        _build(folder, force, verbose)
    return LIB


def _build(folder, force, verbose):
    flags, objects, running, start = nvcc_flags(), [], [], time.time()
    try:
        for s in SOURCES:
            src, obj = os.path.join(CSRC, s), os.path.join(folder, s.replace(".cu", ".o"))
            objects.append(obj)
            if not force and os.path.exists(obj) and os.path.getmtime(obj) >= _newest(_dependencies() + [src]):
                continue
            cmd = flags + ["-c", src, "-o", obj + ".tmp"]
            if verbose:
                print(" ".join(cmd), file=sys.stderr)
            running.append((cmd, obj, subprocess.Popen(cmd)))
        for cmd, obj, p in running:
            if p.wait() != 0:
                raise subprocess.CalledProcessError(p.returncode, cmd)
            _put(obj + ".tmp", obj, start)
    finally:
        for _, obj, p in running:   # the others of a compile that failed
            if p.poll() is None:
                p.terminate()
                p.wait()
            if os.path.exists(obj + ".tmp"):
                os.remove(obj + ".tmp")
    cmd = flags + ["-shared", "-o", LIB + ".tmp"] + objects
    if verbose:
        print(" ".join(cmd), file=sys.stderr)
    subprocess.run(cmd, check=True)
    _put(LIB + ".tmp", LIB, start)
    with open(os.path.join(OBJECTS, "tag"), "w") as f:
        f.write(_tag())


if __name__ == "__main__":
    build(force="--force" in sys.argv)

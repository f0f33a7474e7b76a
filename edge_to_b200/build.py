"""Build libedge_b200.so in-tree with nvcc for sm_100a.

    python -m edge_to_b200.build          (or edge_to_b200.build.build())

The library is a plain C-ABI shared object (include/edge_b200.h) with the CUDA runtime
linked statically, so it loads next to any PyTorch build without sharing its runtime.
"""
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libedge_b200.so")
OBJDIR = os.path.join(HERE, "_build")
SOURCES = ["solver.cu", "batch.cu", "vtail.cu", "fields.cu"]
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def nvcc_path():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _headers():
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC) if not f.endswith(".cu")] + \
        [os.path.join(ROOT, "include", "edge_b200.h")]


def _older(target, deps):
    """True when target is missing or older than one of deps."""
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def _stale():
    return _older(LIB, [os.path.join(CSRC, s) for s in SOURCES] + _headers())


def build(force=False, verbose=False, extra=()):
    """Compile every stale source to an object (in parallel)
    and link the library."""
    if not force and not _stale():
        return LIB
    os.makedirs(OBJDIR, exist_ok=True)
    flags = ["-O3", "-std=c++17", "-lineinfo", *ARCH, "-Xcompiler", "-fPIC", "-cudart", "static",
             "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "include")]
    jobs, objs = [], []
    for src in SOURCES:
        path, obj = os.path.join(CSRC, src), os.path.join(OBJDIR, src + ".o")
        objs.append(obj)
        if force or extra or _older(obj, [path] + _headers()):
            cmd = [nvcc_path(), "-c", *flags, *extra, "-o", obj + ".tmp", path]
            if verbose:
                print(" ".join(cmd), flush=True)
            jobs.append((obj, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for obj, job in jobs:
        out, _ = job.communicate()
        if job.returncode != 0:
            failed = True
            sys.stderr.write(out)
        else:
            os.replace(obj + ".tmp", obj)
            if verbose and out:
                sys.stderr.write(out)
    if failed:
        raise RuntimeError("nvcc failed building libedge_b200.so")
    r = subprocess.run([nvcc_path(), *ARCH, "-shared", "-cudart", "static", "-o", LIB + ".tmp", *objs],
                       capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("nvcc failed linking libedge_b200.so")
    os.replace(LIB + ".tmp", LIB)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True,
          extra=["-Xptxas", "-v"] if "--ptxas" in sys.argv else [])
    print(LIB)

"""Build libmmcuda.so (sm_100a) in-tree with nvcc.

    python micromagnetic.jl_b200/build.py [--force] [-j N]

Sources: micromagnetic.jl_b200/csrc/*.cu; output: micromagnetic.jl_b200/mmcuda/libmmcuda.so.
"""
import argparse
import concurrent.futures
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT_DIR = os.path.join(HERE, "mmcuda")
OBJ_DIR = os.path.join(HERE, "_build")
LIB = os.path.join(OUT_DIR, "libmmcuda.so")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-std=c++20", "-lineinfo", "-Xcompiler", "-fPIC", "-ccbin", "g++",
         "--expt-relaxed-constexpr", "-I", CSRC, "-I", INCLUDE]


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _deps_mtime():
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(INCLUDE, "mmcuda.h")]
    return max(os.path.getmtime(f) for f in files)


def needs_build():
    return not os.path.exists(LIB) or os.path.getmtime(LIB) < _deps_mtime()


def _compile(src, verbose):
    obj = os.path.join(OBJ_DIR, os.path.basename(src) + ".o")
    cmd = [NVCC, *ARCH, *FLAGS, "-c", src, "-o", obj]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{r.stderr}")
    return obj, r.stderr


def _stale(src):
    """The object of src is missing or older than src or any header."""
    obj = os.path.join(OBJ_DIR, os.path.basename(src) + ".o")
    if not os.path.exists(obj):
        return True
    hdrs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hdrs.append(os.path.join(INCLUDE, "mmcuda.h"))
    return os.path.getmtime(obj) < max(os.path.getmtime(f) for f in [src] + hdrs)


def build(force=False, jobs=os.cpu_count() or 4, verbose=False):
    if not force and not needs_build():
        return LIB
    os.makedirs(OBJ_DIR, exist_ok=True)
    todo = [s for s in sources() if force or verbose or _stale(s)]
    with concurrent.futures.ThreadPoolExecutor(max_workers=jobs) as ex:
        # the film-column and run-time y passes take longest: first
        slow = ("mm_rf_c_", "mm_hot_y")
        todo.sort(key=lambda s: not os.path.basename(s).startswith(slow))
        results = list(ex.map(lambda s: _compile(s, verbose), todo))
    objs = [os.path.join(OBJ_DIR, os.path.basename(s) + ".o") for s in sources()]
    if verbose:
        for _, log in results:
            sys.stderr.write(log)
    tmp = LIB + ".tmp"
    cmd = [NVCC, *ARCH, "-shared", "-o", tmp, *objs, "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stderr}")
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("-j", type=int, default=os.cpu_count() or 4)
    ap.add_argument("-v", action="store_true", help="print ptxas resource usage")
    a = ap.parse_args()
    print(build(force=a.force, jobs=a.j, verbose=a.v))

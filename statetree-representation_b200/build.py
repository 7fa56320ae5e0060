"""Builds libstatetree_b200.so (the C-ABI kernel library) in-tree with nvcc for sm_100a.

    python statetree-representation_b200/build.py [--force]

nvcc cross-compiles without a GPU.  Objects are compiled in parallel and linked into
statetree_b200/libstatetree_b200.so next to the Python package (git-ignored; it travels with the working tree).  Beside it
statetree_b200/_calls.so, the host path of module calls (csrc/py_calls.cpp, C++ against this interpreter's torch).
"""
import glob
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "statetree_b200", "libstatetree_b200.so")
CALLS = os.path.join(HERE, "statetree_b200", "_calls.so")
OBJ = os.path.join(HERE, "build")
CALLS_FOR = os.path.join(OBJ, "_calls.txt")
NVCC_FLAGS = ["-Wno-deprecated-gpu-targets", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
              "--expt-relaxed-constexpr"]


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_library(force=False, verbose=False, defines=(), out=None):
    """defines: extra -D macros (a build with other macros goes to its own `out` path and object directory)"""
    out = out or OUT
    obj_dir = OBJ if not defines else os.path.join(OBJ, "_".join(defines))
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    hdrs = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + \
        glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    os.makedirs(obj_dir, exist_ok=True)
    nvcc = os.environ.get("NVCC", "nvcc")

    def compile_one(src):
        obj = os.path.join(obj_dir, os.path.basename(src)[:-3] + ".o")
        if force or _stale(obj, [src] + hdrs):
            cmd = [nvcc] + NVCC_FLAGS + ["-D" + d for d in defines] + (["-Xptxas", "-v"] if verbose else []) + \
                ["-c", src, "-o", obj]
            r = subprocess.run(cmd, capture_output=True, text=True)
            if r.returncode != 0:
                raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
            if verbose:
                print(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(compile_one, srcs))
    if force or _stale(out, objs):
        subprocess.check_call([nvcc, "-Wno-deprecated-gpu-targets", "-shared", "-o", out] + objs)
    return out


def build_calls(force=False):
    """_calls.so from csrc/py_calls.cpp: compiled again when that file or the C ABI's header is newer, and for another torch or
    Python than it was compiled for (noted in CALLS_FOR)"""
    import torch
    src = os.path.join(CSRC, "py_calls.cpp")
    made_for = f"torch {torch.__version__}, {sysconfig.get_config_var('SOABI')}"
    was_for = None
    if os.path.exists(CALLS_FOR):
        with open(CALLS_FOR) as f:
            was_for = f.read()
    if force or was_for != made_for or _stale(CALLS, [src, os.path.join(HERE, "..", "include", "statetree_b200.h")]):
        root = os.path.dirname(torch.__file__)
        cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
        dirs = [f"{root}/include", f"{root}/include/torch/csrc/api/include", f"{cuda}/include", sysconfig.get_paths()["include"]]
        cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
        cmd += [a for d in dirs for a in ("-isystem", d)] + [src, "-o", CALLS, f"-L{root}/lib"]
        r = subprocess.run(cmd + ["-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda"], capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"{cmd[0]} failed on {src}:\n{r.stdout}\n{r.stderr}")
        os.makedirs(OBJ, exist_ok=True)
        with open(CALLS_FOR, "w") as f:
            f.write(made_for)
    return CALLS


if __name__ == "__main__":
    defs = [a[2:] for a in sys.argv[1:] if a.startswith("-D")]
    outs = [a[6:] for a in sys.argv[1:] if a.startswith("--out=")]
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv, defines=defs, out=outs[0] if outs else None))
    print(build_calls(force="--force" in sys.argv))

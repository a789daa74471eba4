"""Builds ``libsvtad.so`` (the C-ABI CUDA library) in-tree with nvcc for sm_100a, and the Python extension
``_native.so`` over it with g++.

    python -m eccv26_tad_b200.build [--force] [--verbose]

The objects go to ``eccv26_tad_b200/_build/`` and the library next to this file.
"""
import argparse
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(PKG, "_build")
LIB = os.path.join(PKG, "libsvtad.so")
NATIVE = os.path.join(PKG, "_native.so")
SOURCES = ["api.cu", "table.cu", "conv_simt.cu", "conv_f32.cu", "conv_f32_tc.cu", "conv_tc.cu", "conv_tc_hybrid.cu", "conv_tc_pair.cu", "conv_tc_pairs.cu", "plan.cu", "allreduce.cu", "noalloc.cu"]
NVCC_FLAGS = ["-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
              "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]


def _nvcc():
    home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cand = os.path.join(home, "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_library(force=False, verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(os.path.dirname(PKG), "include", "svtad.h"))
    sources = [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]
    jobs = []
    for src in sources:
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJ, src.replace(".cu", ".o"))
        if force or _stale(o, [s] + headers):
            cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0 or verbose:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed for " + cmd[-3])

    with ThreadPoolExecutor(max_workers=4) as ex:
        list(ex.map(run, jobs))
    objs = [os.path.join(OBJ, s.replace(".cu", ".o")) for s in sources]
    if force or jobs or _stale(LIB, objs):
        run([_nvcc(), "-shared", "-o", LIB] + objs + ["-lcudart"])
    return LIB


def build_native(force=False, verbose=False):
    """The Python extension over the library: plain g++ against torch's headers, linked to libsvtad.so beside it."""
    import sysconfig
    from torch.utils import cpp_extension
    src = os.path.join(CSRC, "native.cpp")
    deps = [src, os.path.join(os.path.dirname(PKG), "include", "svtad.h"), torch_version_stamp()]
    if not force and not _stale(NATIVE, deps):
        return NATIVE
    inc = cpp_extension.include_paths("cuda") + [sysconfig.get_paths()["include"]]
    libs = cpp_extension.library_paths("cuda")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(_torch_cxx11_abi())]
    cmd += [a for p in inc for a in ("-isystem", p)] + [src, "-o", NATIVE, "-L" + PKG, "-l:libsvtad.so"]
    cmd += ["-L" + p for p in libs] + ["-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python",
                                       "-lcudart", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0 or verbose:
        sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError("g++ failed for native.cpp")
    return NATIVE


def _torch_cxx11_abi():
    import torch
    return torch.compiled_with_cxx11_abi()


def torch_version_stamp():
    """A file that is rewritten when torch changes: the extension is bound to the torch it was compiled against."""
    import torch
    path = os.path.join(OBJ, "torch_version")
    os.makedirs(OBJ, exist_ok=True)
    if not os.path.exists(path) or open(path).read() != torch.__version__:
        with open(path, "w") as f:
            f.write(torch.__version__)
    return path


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build_library(a.force, a.verbose))
    print(build_native(a.force, a.verbose))

"""Builds libvlb.so, the C-ABI engine, for sm_100a with nvcc, and _hostpath.so, the native host side of nn.py, with g++.

Both shared libraries are written next to this file (in-tree) so that they travel
with the source tree; they are never installed into site-packages.  There is no
fallback of any kind: if nvcc fails, building fails.
"""
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libvlb.so")
HOST = os.path.join(HERE, "_hostpath.so")

SOURCES = ["ctx.cu", "elementwise.cu", "normalize.cu", "pool.cu", "bnorm.cu", "roipool.cu", "sampler.cu", "reduce.cu", "fc_small.cu",
           "conv.cu", "conv_simt.cu", "conv_small.cu", "conv_tc.cu", "conv_half.cu"]

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-Xptxas", "-v"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    return "nvcc"


def _deps(src):
    deps = [os.path.join(CSRC, src)]
    deps += [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    deps.append(os.path.join(HERE, "..", "include", "vlb.h"))
    return deps


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def _compile(src, verbose):
    obj = os.path.join(OBJ, src.replace(".cu", ".o"))
    if not _stale(obj, _deps(src)):
        return obj, ""
    cmd = [_nvcc()] + NVCC_FLAGS + ["-c", os.path.join(CSRC, src), "-o", obj]
    p = subprocess.run(cmd, capture_output=True, text=True)
    if p.returncode != 0:
        raise RuntimeError("nvcc failed for %s:\n%s\n%s" % (src, p.stdout, p.stderr))
    log = p.stdout + p.stderr
    with open(obj + ".ptxas.log", "w") as fh:
        fh.write(log)
    return obj, log


def _build_hostpath(force):
    """The CPython module of csrc/hostpath.cpp: torch's C++ API for the tensors, libvlb.so (found beside it) for the work."""
    src = os.path.join(CSRC, "hostpath.cpp")
    if not force and not _stale(HOST, [src, os.path.join(HERE, "..", "include", "vlb.h")]):
        return HOST
    import sysconfig
    import torch
    root = os.path.dirname(os.path.abspath(torch.__file__))
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")]
    lib = os.path.join(root, "lib")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wno-attributes",
           "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI), src, "-o", HOST]
    cmd += [f for d in inc for f in ("-isystem", d)]
    cmd += ["-L" + lib, "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10_cuda", "-lc10", "-L" + HERE, "-l:libvlb.so",
            "-Wl,-rpath," + "$ORIGIN", "-Wl,-rpath," + lib]
    p = subprocess.run(cmd, capture_output=True, text=True)
    if p.returncode != 0:
        raise RuntimeError("g++ failed for hostpath.cpp:\n%s\n%s" % (p.stdout, p.stderr))
    return HOST


def build(force=False, verbose=False):
    """Compile every CUDA source for sm_100a and link libvlb.so, then the host module; returns the library's path."""
    os.makedirs(OBJ, exist_ok=True)
    if force:
        for f in os.listdir(OBJ):
            if f.endswith(".o"):
                os.remove(os.path.join(OBJ, f))
    with ThreadPoolExecutor(max_workers=min(8, len(SOURCES))) as ex:
        results = list(ex.map(lambda s: _compile(s, verbose), SOURCES))
    objs = [r[0] for r in results]
    if verbose:
        for _, log in results:
            if log:
                sys.stderr.write(log)
    if force or _stale(LIB, objs):
        cmd = [_nvcc(), "-shared", "-o", LIB] + objs + ["-lcudart"]
        p = subprocess.run(cmd, capture_output=True, text=True)
        if p.returncode != 0:
            raise RuntimeError("link failed:\n%s\n%s" % (p.stdout, p.stderr))
    _build_hostpath(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))

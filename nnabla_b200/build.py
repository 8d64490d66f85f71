"""Builds nnabla_b200/lib/libnnabla_b200.so from nnabla_b200/csrc/*.cu with nvcc for
sm_100a (cross-compiles without a GPU), and nnabla_b200/lib/_native.so, its binding to torch
tensors, from csrc/native.cpp. Usage: python -m nnabla_b200.build [--force] [-v]"""
import concurrent.futures
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIBDIR = os.path.join(HERE, "lib")
OBJDIR = os.path.join(ROOT, "build", "nnabla_b200")
LIB = os.path.join(LIBDIR, "libnnabla_b200.so")
NATIVE = os.path.join(LIBDIR, "_native.so")

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I" + os.path.join(ROOT, "include"), "-I" + CSRC]


def nvcc():
    for c in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if c and os.path.exists(c):
            return c
    raise RuntimeError("nvcc not found")


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _newest_header():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs.append(os.path.join(ROOT, "include", "nnabla_b200.h"))
    return max(os.path.getmtime(h) for h in hs)


def build(force=False, verbose=False):
    os.makedirs(LIBDIR, exist_ok=True)
    os.makedirs(OBJDIR, exist_ok=True)
    cc = nvcc()
    hdr = _newest_header()
    jobs = []
    objs = []
    for src in _sources():
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJDIR, src[:-3] + ".o")
        objs.append(o)
        if force or not os.path.exists(o) or os.path.getmtime(o) < max(os.path.getmtime(s), hdr):
            cmd = [cc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    with concurrent.futures.ThreadPoolExecutor(max_workers=8) as ex:
        for cmd, r in ex.map(run, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(" ".join(cmd[-3:]) + "\n" + r.stdout + r.stderr)
            if r.returncode != 0:
                raise RuntimeError("nvcc failed for " + cmd[-3])
    if jobs or force or not os.path.exists(LIB):
        cmd = [cc, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-lpthread", "-ldl"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    _build_native(force)
    return LIB


def _build_native(force):
    src = os.path.join(CSRC, "native.cpp")
    newest = max(os.path.getmtime(src), os.path.getmtime(os.path.join(ROOT, "include", "nnabla_b200.h")))
    if not force and os.path.exists(NATIVE) and os.path.getmtime(NATIVE) >= newest:
        return
    import sysconfig

    import torch
    base = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc())))
    include = [os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"),
               os.path.join(cuda, "include"), sysconfig.get_paths()["include"], os.path.join(ROOT, "include")]
    libs = ["torch_python", "torch", "torch_cuda", "torch_cpu", "c10", "c10_cuda"]
    cmd = (["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", NATIVE, src,
            "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI)] + ["-I" + d for d in include] +
           ["-L" + os.path.join(base, "lib")] + ["-l" + n for n in libs] +
           ["-L" + LIBDIR, "-lnnabla_b200", "-Wl,-rpath,$ORIGIN"])
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("g++ failed for " + src)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))

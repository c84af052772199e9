"""Build libwinograd2x2_b200.so in this directory with nvcc for sm_100a, and wg2x2/_native.so, the Python calls over it.

Usage: python build.py [--force] [--verbose]
"""
import importlib.util
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
SOURCES = ["imtrans.cu", "conv_ffma.cu", "conv_tc.cu", "api.cu", "ref_launchers.cu", "noalloc.cu", "pool.cu"]
LIB = os.path.join(HERE, "libwinograd2x2_b200.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
NATIVE = os.path.join(HERE, "wg2x2", "_native.so")
BINDINGS = os.path.join(CSRC, "bindings.cpp")
CXX = os.environ.get("CXX", "g++")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
         "-Xcompiler", "-fPIC", "-DWG2X2_BUILD"]


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _start_bindings():
    """Compile wg2x2/_native.so against the installed torch's headers and libraries (both found without importing torch)."""
    torch = importlib.util.find_spec("torch").submodule_search_locations[0]
    cuda = os.path.dirname(os.path.dirname(NVCC))
    inc = [os.path.join(torch, "include"), os.path.join(torch, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    cmd = [CXX, "-O2", "-std=c++17", "-fPIC", "-c", BINDINGS, "-o", os.path.join(HERE, "build", "bindings.o")]
    for d in inc:
        cmd += ["-isystem", d]
    link = [CXX, "-shared", "-o", NATIVE, os.path.join(HERE, "build", "bindings.o"), "-L" + HERE, "-lwinograd2x2_b200",
            "-Wl,-rpath,$ORIGIN/..", "-L" + os.path.join(torch, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda",
            "-lc10", "-lc10_cuda"]
    return subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True), link


def build(force=False, verbose=False):
    header = os.path.join(HERE, "..", "include", "winograd2x2_b200.h")
    cuda_src = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f != os.path.basename(BINDINGS)] + [header]
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    bindings = _start_bindings() if force or _stale(NATIVE, [BINDINGS, header]) else None
    if force or _stale(LIB, cuda_src):
        objs = []
        procs = []
        for s in SOURCES:
            o = os.path.join(HERE, "build", s.replace(".cu", ".o"))
            cmd = [NVCC] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", os.path.join(CSRC, s), "-o", o]
            procs.append((s, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
            objs.append(o)
        for s, p in procs:
            out, _ = p.communicate()
            if verbose or p.returncode:
                sys.stderr.write(out)
            if p.returncode:
                raise RuntimeError("nvcc failed on " + s)
        subprocess.check_call([NVCC, "-shared", "-o", LIB] + objs + ["-lcudart", "-lcuda"])
    if bindings is not None:
        proc, link = bindings
        out, _ = proc.communicate()
        if verbose or proc.returncode:
            sys.stderr.write(out)
        if proc.returncode:
            raise RuntimeError("%s failed on bindings.cpp" % CXX)
        subprocess.check_call(link)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))

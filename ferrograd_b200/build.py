"""Builds libferrograd_b200.so in-tree with nvcc for sm_100a, and the CPython module of its frequent entry points.

Usage: python -m ferrograd_b200.build [--force] [--verbose]
"""
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "libferrograd_b200.so")
SOURCES = ["ctx.cu", "optim.cu", "softmax.cu", "eltwise.cu", "gemm_simt.cu", "gemm_fma.cu", "gemm_tc.cu", "mse_noalloc.cu", "graph.cu", "bpat.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "--fmad=false", "-Xcompiler", "-fPIC", "-cudart", "static"]


def _newest(paths):
    return max(os.path.getmtime(p) for p in paths)


CALLS_SRC = os.path.join(CSRC, "calls.cpp")
CALLS = os.path.join(HERE, "_calls" + sysconfig.get_config_var("EXT_SUFFIX"))


def build_calls(force: bool = False) -> None:
    """The module of frequent entry points (csrc/calls.cpp), beside the library that it calls."""
    header = os.path.join(os.path.dirname(HERE), "include", "ferrograd_b200.h")
    if not force and os.path.exists(CALLS) and os.path.getmtime(CALLS) >= _newest([CALLS_SRC, header]):
        return
    tmp = CALLS + ".tmp"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", sysconfig.get_paths()["include"], CALLS_SRC, "-o", tmp,
                    "-L", HERE, "-lferrograd_b200", "-Wl,-rpath,$ORIGIN"], check=True)
    os.replace(tmp, CALLS)


def build(force: bool = False, verbose: bool = False) -> str:
    out = build_library(force, verbose)
    build_calls(force)
    return out


def build_library(force: bool = False, verbose: bool = False) -> str:
    srcs = [os.path.join(CSRC, s) for s in SOURCES]
    deps = srcs + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    deps.append(os.path.join(os.path.dirname(HERE), "include", "ferrograd_b200.h"))
    if not force and os.path.exists(OUT) and os.path.getmtime(OUT) >= _newest(deps):
        return OUT
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    extra = os.environ.get("FG_NVCC_EXTRA", "").split()      # e.g. -DFG_GEMM_PROFILE for a diagnostic build
    objs = []
    procs = []
    for s in srcs:
        o = s[:-3] + ".o"
        objs.append(o)
        cmd = [nvcc] + NVCC_FLAGS + extra + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
        procs.append((cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for cmd, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            print(out)
        if p.returncode != 0:
            raise RuntimeError("nvcc failed: " + " ".join(cmd))
    # link beside the target and move into place: a reader (a loader, a copy of the tree) sees a whole file
    tmp = OUT + ".tmp"
    link = [nvcc, "-shared", "-cudart", "static", "-o", tmp] + objs + ["-ldl"]
    subprocess.run(link, check=True)
    os.replace(tmp, OUT)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))

"""Builds the native parts of sodecl_b200 in-tree.

Outputs (next to this file):
  libsodecl_cuda.so                 C ABI (include/sodecl_cuda.h), NVRTC front end,
                                    sm_100a helper kernels, C++ sodecl::sodeclmgr
  sodecl_interface<EXT_SUFFIX>      pybind11 module (the reference's Python binding)

Host C++ is compiled by g++, the .cu file by nvcc for sm_100a only
(-gencode arch=compute_100a,code=sm_100a); the solver kernels themselves are
compiled at run time by NVRTC, for sm_100a, from device/*.cuh, which this
script embeds into the library as string constants.
"""
from __future__ import annotations

import hashlib
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(REPO, "include")
OBJ = os.path.join(HERE, "_build")
CUDA_HOME = os.environ.get("CUDA_HOME", "/usr/local/cuda")
NVCC = os.path.join(CUDA_HOME, "bin", "nvcc")
LIB = os.path.join(HERE, "libsodecl_cuda.so")
GENCODE = ["-gencode", "arch=compute_100a,code=sm_100a"]
CUDA_SOURCES = ["aux_kernels.cu", "batch_noalloc.cu"]

EMBED = [("kFastDivSrc", "fastdiv.cuh"), ("kPreludeSrc", "prelude.cuh"), ("kMathCoreSrc", "mathcore.cuh"),
         ("kFastMathSrc", "fastmath.cuh"), ("kThreefrySrc", "threefry.cuh"), ("kSolversSrc", "solvers.cuh"),
         ("kBatchSrc", "batch.cuh"), ("kAdjointSrc", "adjoint.cuh")]


def _run(cmd, verbose):
    if verbose:
        print(" ".join(cmd))
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError("command failed: %s\n%s%s" % (" ".join(cmd), proc.stdout, proc.stderr))
    return proc


def _digest(paths, extra=""):
    h = hashlib.sha256(extra.encode())
    for p in paths:
        h.update(p.encode())
        with open(p, "rb") as f:
            h.update(f.read())
    return h.hexdigest()


def _fresh(target, digest):
    stamp = target + ".stamp"
    return os.path.exists(target) and os.path.exists(stamp) and open(stamp).read() == digest


def _stamp(target, digest):
    with open(target + ".stamp", "w") as f:
        f.write(digest)


def write_embedded():
    """device/*.cuh -> embedded_sources.inc (raw string literals)."""
    out = ["// generated by sodecl_b200/build.py from device/*.cuh -- do not edit\n"]
    for name, fname in EMBED:
        text = open(os.path.join(CSRC, "device", fname)).read()
        delim = "SODECL_SRC"
        assert (")" + delim + '"') not in text
        # raw literals have a length limit on some compilers; split into pieces
        pieces = [text[i:i + 8000] for i in range(0, len(text), 8000)] or [""]
        out.append("const char %s[] =\n" % name)
        for p in pieces:
            out.append('R"%s(%s)%s"\n' % (delim, p, delim))
        out.append(";\n")
    path = os.path.join(CSRC, "embedded_sources.inc")
    content = "".join(out)
    if not os.path.exists(path) or open(path).read() != content:
        with open(path, "w") as f:
            f.write(content)
    return path


def build(verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    write_embedded()
    cxxflags = ["-O2", "-fPIC", "-std=c++17", "-Wall", "-Wno-unused-function", "-I", INCLUDE, "-I", CSRC,
                "-I", os.path.join(CUDA_HOME, "include")]
    objects = []
    headers = [os.path.join(INCLUDE, h) for h in os.listdir(INCLUDE)] + \
              [os.path.join(CSRC, h) for h in os.listdir(CSRC) if h.endswith((".hpp", ".inc"))] + \
              [os.path.join(CSRC, "device", h) for h in os.listdir(os.path.join(CSRC, "device"))]
    for src in ("program.cpp", "speculable.cpp", "sodecl_cuda.cpp", "batch.cpp", "sodeclmgr.cpp"):
        obj = os.path.join(OBJ, src + ".o")
        cmd = ["g++"] + cxxflags + ["-c", os.path.join(CSRC, src), "-o", obj]
        d = _digest([os.path.join(CSRC, src)] + sorted(headers), " ".join(cmd))
        if not _fresh(obj, d):
            _run(cmd, verbose)
            _stamp(obj, d)
        objects.append(obj)
    for name in CUDA_SOURCES:
        cu = os.path.join(CSRC, name)
        obj = os.path.join(OBJ, name + ".o")
        cmd = [NVCC] + GENCODE + ["-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-I", INCLUDE, "-I", CSRC,
                                  "-c", cu, "-o", obj]
        d = _digest([cu] + sorted(headers), " ".join(cmd))
        if not _fresh(obj, d):
            _run(cmd, verbose)
            _stamp(obj, d)
        objects.append(obj)

    libdir = os.path.join(CUDA_HOME, "lib64")
    link = ["g++", "-shared", "-o", LIB] + objects + [
        "-L", libdir, "-lcudart_static", "-lnvrtc", "-ldl", "-lpthread", "-lrt",
        "-Wl,-rpath," + libdir, "-Wl,--no-undefined", "-Wl,-soname,libsodecl_cuda.so"]
    d = _digest(objects, " ".join(link))
    if not _fresh(LIB, d):
        _run(link, verbose)
        _stamp(LIB, d)

    build_python_module(verbose)
    return LIB


def python_module_path():
    return os.path.join(HERE, "sodecl_interface" + sysconfig.get_config_var("EXT_SUFFIX"))


def build_python_module(verbose=False):
    import pybind11

    target = python_module_path()
    src = os.path.join(CSRC, "pybind_module.cpp")
    cmd = ["g++", "-O2", "-fPIC", "-shared", "-std=c++17", "-I", INCLUDE, "-I", pybind11.get_include(),
           "-I", sysconfig.get_paths()["include"], src, "-o", target, "-L", HERE, "-lsodecl_cuda",
           "-Wl,-rpath,$ORIGIN"]
    d = _digest([src, os.path.join(INCLUDE, "sodeclmgr.hpp"), os.path.join(INCLUDE, "sodecl_cuda.h"), LIB],
                " ".join(cmd))
    if not _fresh(target, d):
        _run(cmd, verbose)
        _stamp(target, d)
    return target


if __name__ == "__main__":
    build(verbose="-v" in sys.argv)
    print("built", LIB)

"""csrc/device's elementary functions and quotients compiled for the host (cpp/device_math.cpp)."""
import ctypes
import functools
import os
import subprocess
import tempfile

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "sodecl_b200", "csrc")


@functools.lru_cache(maxsize=1)
def library():
    so = os.path.join(tempfile.mkdtemp(), "device_math.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC,
                    os.path.join(HERE, "cpp", "device_math.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def call(name, *arrays):
    """Runs the array function `name` on arrays of one length (the last ones are its outputs)."""
    getattr(library(), name)(*(ctypes.c_void_p(a.ctypes.data) for a in arrays), ctypes.c_long(arrays[0].size))


def values(fn, x):
    y = np.empty_like(x)
    call(fn + "_values", x, y)
    return y


def ulps(got, want):
    """|got - want| in units of want's last place, want in long double."""
    exponent = np.maximum(np.frexp(np.abs(want))[1] - 53, -1074)
    return (np.abs(got - want) / np.ldexp(np.longdouble(1), exponent)).astype(np.float64)

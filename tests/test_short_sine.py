"""The short sine and cosine of the fp32 network (``sincos_short``, landmark_b200/csrc/gnr_split.cuh), compiled for the host
from its source and compared with fp64: the errors its comment states, over the range it is used in."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HOST = """
#include <math.h>
#include <string.h>
#define __device__
#define __forceinline__ static inline
static inline int __float_as_int(float x) { int i; memcpy(&i, &x, 4); return i; }
static inline float __int_as_float(int i) { float x; memcpy(&x, &i, 4); return x; }
%s
extern "C" void run(const float* x, float* s, float* c, long n) { for (long i = 0; i < n; ++i) sincos_short(x[i], s[i], c[i]); }
"""


@pytest.fixture(scope="module")
def short_sine(tmp_path_factory):
    text = open(os.path.join(ROOT, "landmark_b200", "csrc", "gnr_split.cuh")).read()
    beg = text.index("__device__ __forceinline__ void sincos_short")
    folder = tmp_path_factory.mktemp("sine")
    src, lib = folder / "sine.cpp", folder / "sine.so"
    src.write_text(HOST % text[beg:text.index("\n}\n", beg) + 3])
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", str(src), "-o", str(lib)], check=True)
    run = C.CDLL(str(lib)).run
    run.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_long]

    def call(x):
        s, c = np.empty_like(x), np.empty_like(x)
        run(x.ctypes.data, s.ctypes.data, c.ctypes.data, x.size)
        return s.astype(np.float64), c.astype(np.float64)

    return call


@pytest.mark.parametrize("span", [1e-3, 0.5, 2.0, 30.0, 1000.0])
def test_errors_are_what_the_comment_states(short_sine, span):
    rng = np.random.RandomState(int(span * 1000) + 1)
    x = np.concatenate([rng.uniform(-span, span, 2000000), [0.0, -0.0, span, -span]]).astype(np.float32)
    quarter = np.round(x[:200000].astype(np.float64) / (np.pi / 4)) * (np.pi / 4)  # and around the ends of the quadrants
    near = quarter.astype(np.float32)
    x = np.concatenate([x, near, np.nextafter(near, np.float32(2e3)), np.nextafter(near, np.float32(-2e3))])
    x = x[np.abs(x) <= 1000.0]
    s, c = short_sine(x)
    err = np.stack([s - np.sin(x.astype(np.float64)), c - np.cos(x.astype(np.float64))])
    assert np.abs(err).max() <= 7.1e-8, np.abs(err).max()
    assert np.sqrt((err ** 2).mean()) <= 1.7e-8, np.sqrt((err ** 2).mean())

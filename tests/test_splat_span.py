"""The density splat's voxel span of a particle along one axis (splat_box.h), compiled for the host: positions that no
tank produces (infinite or beyond the integers) have an empty span, NaN (which fails every distance test) at most one
voxel, and every other position the span of the reference's rounding in integers without a limit."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

from slosh_b200 import build

SOURCE = """
#include "splat_box.h"
extern "C" void span(float c, float rr, int n, int whole, int* out) {
    const slosh::SplatSpan s = slosh::splat_span(c, rr, n, whole != 0);
    out[0] = s.lo;
    out[1] = s.hi;
}
"""


@pytest.fixture(scope="module")
def span(tmp_path_factory):
    d = tmp_path_factory.mktemp("splat_span")
    (d / "span.cpp").write_text(SOURCE)
    lib = str(d / "span.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fwrapv", "-shared", "-fPIC", "-I", os.path.join(build.HERE, "csrc"),
                    str(d / "span.cpp"), "-o", lib], check=True)
    f = C.CDLL(lib).span
    f.argtypes = [C.c_float, C.c_float, C.c_int, C.c_int, C.POINTER(C.c_int)]

    def call(c, rr, n, whole):
        out = (C.c_int * 2)()
        f(c, rr, n, int(whole), out)
        return out[0], out[1]

    return call


def _expected(c, rr, n, whole):
    f = np.float32
    c, rr = f(c), f(rr)
    lo, hi = max(math.floor((c - rr) - f(0.5)), 0), min(math.ceil((c + rr) - f(0.5)), n - 1)
    if lo > hi:
        return None
    if whole:
        far = rr * f(1.001)
        lo += int((f(lo) + f(0.5)) - c < -far)
        hi -= int((f(hi) + f(0.5)) - c > far)
    return (lo, hi) if lo <= hi else None


# kernels of the default size, cut by the footprint, and wide enough for the general voxel loop
@pytest.mark.parametrize("rr,whole", [(1.2, True), (0.3, True), (2.7, True), (4.0, False), (4.0, True)])
@pytest.mark.parametrize("n", [1, 8, 24, 4096])
def test_span(span, rr, whole, n):
    far = [math.inf, -math.inf, math.nan, 1e30, -1e30, 3.4e38, -3.4e38]
    far += [s * v for s in (1.0, -1.0) for v in (2.0 ** 31, 2.0 ** 31 - 128.0, 2.0 ** 31 + 256.0, 2.0 ** 30, 1e9)]
    for c in far:
        lo, hi = span(c, rr, n, whole)
        assert lo > hi or (math.isnan(c) and (lo, hi) == (0, 0)), (c, lo, hi)
    rng = np.random.default_rng(n)
    near = np.concatenate([rng.uniform(-8.0, n + 8.0, 4000), np.arange(-6, min(n, 64) + 6) + 0.5, np.arange(-6, min(n, 64) + 6),
                           [-0.0, -rr, rr, n - rr, n + rr, n + rr + 0.5, -rr - 0.5]])
    for c in near.astype(np.float32):
        lo, hi = span(float(c), rr, n, whole)
        want = _expected(c, rr, n, whole)
        assert (lo, hi) == want if want else lo > hi, (c, lo, hi, want)

"""The solver's quotient from a stored reciprocal (exact_div.h) against division, bit for bit: on the host and, compiled with
the library's flags, on the GPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from slosh_b200 import build

HOST = """
#include "exact_div.h"
extern "C" void quotients(const float* a, const float* d, float* q, int n) {
    for (int i = 0; i < n; ++i) q[i] = slosh::div_by(a[i], d[i], 1.0f / d[i]);
}
"""
DEVICE = """
#include "exact_div.h"
__global__ void k(const float* a, const float* d, float* q, float* r, int n) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    q[i] = slosh::div_by(a[i], d[i], 1.0f / d[i]);
    r[i] = a[i] / d[i];
}
extern "C" __attribute__((visibility("default"))) int quotients(const float* a, const float* d, float* q, float* r, int n) {
    k<<<(n + 255) / 256, 256>>>(a, d, q, r, n);
    return int(cudaDeviceSynchronize());
}
"""


def _pairs():
    """Numerators of every exponent, the ends of the corrected range and what has no value; the diagonals of a coarse level
    (epsilon and up to six neighbours), of free surfaces (theta down to 0.05) and any between."""
    rng = np.random.default_rng(11)
    n = 1 << 20
    any_bits = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32).view(np.float32)
    usual = (rng.standard_normal(n) * 10.0 ** rng.uniform(-12, 12, n)).astype(np.float32)
    ends = np.float32([1e-25, 1e25])
    steps = (ends.view(np.int32)[:, None] + np.arange(-64, 65, dtype=np.int32)).reshape(-1).view(np.float32)
    special = np.float32([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-45, -1e-45, 1.17549435e-38, 3.4028235e38, -3.4028235e38, 1.0, -1.0])
    a = np.concatenate([any_bits, usual, steps, -steps, special])
    eps = np.float32(1e-4)
    levels = [eps]
    for _ in range(6):
        levels.append(np.float32(levels[-1] + np.float32(1.0)))
    surface = (eps + np.float32(5.0) + np.float32(1.0) / rng.uniform(0.05, 1.0, 4096).astype(np.float32)).astype(np.float32)
    spread = (10.0 ** rng.uniform(-4, 3, 4096)).astype(np.float32)
    d = np.concatenate([np.tile(np.float32(levels), 1200), surface, spread])
    out_a = np.concatenate([a, np.repeat(np.concatenate([steps, -steps, special]), len(levels))])
    out_d = np.concatenate([rng.choice(d, len(a)), np.tile(np.float32(levels), 2 * len(steps) + len(special))])
    return np.ascontiguousarray(out_a), np.ascontiguousarray(out_d)


def _same(q, want):
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(q), nan)
    assert np.array_equal(q[~nan].view(np.uint32), want[~nan].view(np.uint32))


def test_quotients_on_the_host(tmp_path):
    (tmp_path / "q.cpp").write_text(HOST)
    lib = str(tmp_path / "q.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", os.path.join(build.HERE, "csrc"),
                    str(tmp_path / "q.cpp"), "-o", lib], check=True)
    a, d = _pairs()
    q = np.empty_like(a)
    C.CDLL(lib).quotients(*[v.ctypes.data_as(C.c_void_p) for v in (a, d, q)], C.c_int(len(a)))
    with np.errstate(all="ignore"):
        _same(q, a / d)


@pytest.mark.gpu
def test_quotients_on_the_gpu(tmp_path):
    import torch

    (tmp_path / "q.cu").write_text(DEVICE)
    lib = str(tmp_path / "q.so")
    subprocess.run([build.NVCC] + build.FLAGS + ["-shared", "-I", os.path.join(build.HERE, "csrc"), str(tmp_path / "q.cu"), "-o", lib,
                                                 "-lcudart"], check=True)
    a, d = _pairs()
    ta, td = torch.from_numpy(a).cuda(), torch.from_numpy(d).cuda()
    q, r = torch.empty_like(ta), torch.empty_like(ta)
    torch.cuda.synchronize()
    assert C.CDLL(lib).quotients(*[C.c_void_p(t.data_ptr()) for t in (ta, td, q, r)], C.c_int(len(a))) == 0
    _same(q.cpu().numpy(), r.cpu().numpy())
    with np.errstate(all="ignore"):
        _same(r.cpu().numpy(), a / d)

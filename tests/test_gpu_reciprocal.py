"""GPU: the sparse factorization's reciprocal (csrc/mp_recip.cuh) against 1/d in 80-bit
arithmetic, over random mantissas and exponents and at the ends of its range, and
the range itself.

Bound: the last rounding, 2^-53 relative, and 2^-60 that the iteration leaves out
(the third power of the approximation's 2^-20), with room for the two inner
roundings: 2^-53 (1 + 2^-6)."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from minipic_b200.build import ARCH, CSRC, _nvcc

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include "mp_recip.cuh"
__global__ void k(int n, const double *d, double *r, int *ok) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    r[i] = mp::reciprocal(d[i]);
    ok[i] = mp::invertible(d[i]);
}
extern "C" int run(int n, const double *d, double *r, int *ok) {
    double *a = nullptr, *b = nullptr;
    int *c = nullptr;
    cudaMalloc(&a, 8 * (size_t)n);
    cudaMalloc(&b, 8 * (size_t)n);
    cudaMalloc(&c, 4 * (size_t)n);
    if (!a || !b || !c) return -1;
    cudaMemcpy(a, d, 8 * (size_t)n, cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(n, a, b, c);
    cudaMemcpy(r, b, 8 * (size_t)n, cudaMemcpyDeviceToHost);
    cudaMemcpy(ok, c, 4 * (size_t)n, cudaMemcpyDeviceToHost);
    cudaFree(a);
    cudaFree(b);
    cudaFree(c);
    return cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("recip")
    src, lib = str(d / "r.cu"), str(d / "r.so")
    with open(src, "w") as f:
        f.write(PROGRAM)
    subprocess.run([_nvcc(), *ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", CSRC, src, "-o", lib],
                   check=True)
    L = ctypes.CDLL(lib)

    def call(x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        r, ok = np.zeros_like(x), np.zeros(x.size, dtype=np.int32)
        p = ctypes.c_void_p
        assert L.run(x.size, x.ctypes.data_as(p), r.ctypes.data_as(p), ok.ctypes.data_as(p)) == 0
        return r, ok != 0

    return call


def test_against_80_bits(run):
    rng = np.random.default_rng(0)
    m = np.concatenate([rng.uniform(1.0, 2.0, 1 << 20), 1.0 + np.arange(4096) * 2.0 ** -52,
                        2.0 - np.arange(1, 4097) * 2.0 ** -52, 1.0 + np.arange(1 << 16) * 2.0 ** -16])
    for e in (rng.integers(-960, 961, m.size), np.zeros(m.size, int), np.full(m.size, -960), np.full(m.size, 960)):
        d = np.ldexp(m, e) * rng.choice((-1.0, 1.0), m.size)
        r, ok = run(d)
        assert ok.all()
        err = np.abs(r.astype(np.longdouble) * d.astype(np.longdouble) - 1)
        assert err.max() <= 2.0 ** -53 * (1 + 2.0 ** -6), float(err.max() * 2.0 ** 53)


def test_range(run):
    lo, hi = 2.0 ** -960, 2.0 ** 961
    inside = np.array([lo, np.nextafter(hi, 0), 1.0, 1e-280, 1e280])
    outside = np.array([0.0, np.nextafter(lo, 0), hi, 5e-324, 1e-300, 1e300, np.inf, np.nan])
    for s in (1.0, -1.0):
        assert run(s * inside)[1].all()
        assert not run(s * outside)[1].any()

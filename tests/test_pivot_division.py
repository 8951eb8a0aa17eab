"""Division by a pivot through its reciprocal (csrc/radm2_div.cuh): the bits of a / u, signs of
zeros among them, over the whole exponent range.

The header is compiled for the host, where the product, the fused multiply-add and the division
are IEEE's too, and on the GPU with nvcc against CUDA's own division.
"""
import ctypes
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG

CSRC = os.path.join(PKG, "csrc")

HOST = '''
#include <cmath>
#include <cstdint>
#include <cstring>
using std::fma;
#define __device__
#define __forceinline__ inline
#define __noinline__
static int __double2hiint(double x) { int64_t v; std::memcpy(&v, &x, 8); return (int)(v >> 32); }
static double __hiloint2double(int h, int l) { int64_t v = ((int64_t)h << 32) | (uint32_t)l; double x; std::memcpy(&x, &v, 8); return x; }
static double __drcp_rn(double x) { return 1.0 / x; }
static int __any_sync(unsigned, int p) { return p; }
#include "radm2_div.cuh"
extern "C" int quotients(long n, const double *a, const double *u, double *q, double *plain)
{
    for (long i = 0; i < n; i++) {
        q[i] = radm2::div_pivot(a[i], u[i], radm2::rcp_pivot(u[i]));
        plain[i] = a[i] / u[i];
    }
    return 0;
}
'''

DEVICE = '''
#include "radm2_div.cuh"
__global__ void k(long n, const double *a, const double *u, double *q, double *plain)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        q[i] = radm2::div_pivot(a[i], u[i], radm2::rcp_pivot(u[i]));
        plain[i] = a[i] / u[i];
    }
}
extern "C" int quotients(long n, const double *a, const double *u, double *q, double *plain)
{
    if (n % 32) return -1;  // whole warps: div_pivot is called by all lanes together
    double *d = nullptr;
    if (cudaMalloc(&d, 32 * n) != cudaSuccess) return -2;
    cudaMemcpy(d, a, 8 * n, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, u, 8 * n, cudaMemcpyHostToDevice);
    k<<<296, 256>>>(n, d, d + n, d + 2 * n, d + 3 * n);
    cudaMemcpy(q, d + 2 * n, 8 * n, cudaMemcpyDeviceToHost);
    const cudaError_t e = cudaMemcpy(plain, d + 3 * n, 8 * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : -3;
}
'''


def _pairs(m, seed):
    """Numerators and pivots: random mantissas over all exponents, over the exponents of real
    factorisations, quotients next to a rounding boundary, and the special values crossed."""
    r = np.random.RandomState(seed)

    def rand(lo, hi):
        x = np.ldexp(1.0 + r.randint(0, 1 << 52, m, dtype=np.int64) / 2.0**52, r.randint(lo, hi, m))
        return np.where(r.rand(m) < 0.5, -x, x)
    a = [rand(-1080, 1024), rand(-40, 40), rand(-1074, -960), rand(-1022, 1023)]
    u = [rand(-1080, 1024), rand(-30, 30), rand(60, 105), rand(-105, 105)]
    # a = u (q + ulp / 2), rounded: the quotient lies next to the middle of two neighbours
    v, q = rand(-20, 20), rand(-20, 20)
    a.append(v * q + v * np.spacing(q) * 0.5)
    u.append(v)
    tiny = np.finfo(float).tiny
    s = np.array([0.0, -0.0, 1.0, -1.0, 3.0, 5e-324, -5e-324, tiny, 2.0**-100, 2.0**100, -2.0**100, 2.0**101, 2.0**-101, 1e300, -1e300,
                  np.finfo(float).max, np.inf, -np.inf, np.nan, 2.0**-975, 2.0**-1000, 1.5 * 2.0**75, 7.0e5, -7.0e5])
    g = np.meshgrid(s, s)
    a, u = np.concatenate(a + [g[0].ravel()]), np.concatenate(u + [g[1].ravel()])
    n = len(a) // 32 * 32 + 32
    return np.resize(a, n), np.resize(u, n)


def _check(lib, a, u):
    lib.quotients.argtypes = [ctypes.c_long] + [ctypes.c_void_p] * 4
    q, p = np.empty_like(a), np.empty_like(a)
    assert lib.quotients(len(a), *(x.ctypes.data for x in (a, u, q, p))) == 0
    same = (q.view(np.int64) == p.view(np.int64)) | (np.isnan(q) & np.isnan(p))
    bad = np.flatnonzero(~same)
    assert len(bad) == 0, [(float(a[i]).hex(), float(u[i]).hex(), float(q[i]).hex(), float(p[i]).hex()) for i in bad[:5]]
    return p


def test_quotients_on_the_host(tmp_path):
    src, so = tmp_path / "div.cpp", tmp_path / "div.so"
    src.write_text(HOST)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, str(src), "-o", str(so)], check=True)
    a, u = _pairs(300000, 1)
    with np.errstate(all="ignore"):
        p = _check(ctypes.CDLL(str(so)), a, u)
        assert np.array_equal(p, a / u, equal_nan=True)


def test_no_reciprocal_estimates():
    """Reciprocals and divisions come from CUDA's functions, not from the hardware's estimates."""
    for name in os.listdir(CSRC):
        if name.endswith((".cu", ".cuh", ".h")):
            assert not re.search(r"\b(rcp|div|rsqrt|sqrt|ex2|lg2)\.approx", open(os.path.join(CSRC, name)).read()), name


@pytest.mark.gpu
def test_quotients_on_the_gpu(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, so = tmp_path / "div.cu", tmp_path / "div.so"
    src.write_text(DEVICE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "--fmad=false", "-Xcompiler", "-fPIC", "-shared", "-I", CSRC,
                    str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    for seed in range(4):
        _check(lib, *_pairs(2000000, seed))

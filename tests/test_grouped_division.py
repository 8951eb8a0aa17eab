"""Four quotients with one division (div_four in csrc/radm2_div.cuh).

The corrected quotient is within 2^-47 ulp of the exact one before its last rounding.  So it has the
bits of a / u unless the quotient lies that close to the middle of two neighbours: of 2^23 random
quotients none is expected to differ (chance 1e-7), and next to a middle the two are neighbours.
Compiled for the host, where the operations are IEEE's too, and on the GPU against CUDA's division.
"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG
from test_pivot_division import HOST

CSRC = os.path.join(PKG, "csrc")

BODY = '''
        double q4[4];
        const double a4[4] = {a[i], a[i + 1], a[i + 2], a[i + 3]}, u4[4] = {u[i], u[i + 1], u[i + 2], u[i + 3]};
        radm2::div_four(a4, u4, q4);
        for (int j = 0; j < 4; j++) {
            q[i + j] = q4[j];
            plain[i + j] = a[i + j] / u[i + j];
        }
'''

DEVICE = '''
#include "radm2_div.cuh"
__global__ void k(long n, const double *a, const double *u, double *q, double *plain)
{
    for (long i = 4 * (blockIdx.x * (long)blockDim.x + threadIdx.x); i < n; i += 4 * (long)gridDim.x * blockDim.x) {
''' + BODY + '''
    }
}
extern "C" int grouped(long n, const double *a, const double *u, double *q, double *plain)
{
    if (n % 4) return -1;
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


def _random(m, seed):
    """Squares of errors and scales: over the exponents they have, over the whole range, and with
    zeros, infinities, NaN and subnormals among them."""
    r = np.random.RandomState(seed)

    def rand(lo, hi):
        return np.ldexp(1.0 + r.randint(0, 1 << 52, m, dtype=np.int64) / 2.0**52, r.randint(lo, hi, m))
    a = [rand(-80, 60), rand(-80, 60), rand(-1074, 1024), rand(-705, 705)]
    u = [rand(-20, 60), rand(-205, 205), rand(-1074, 1024), rand(-199, 199)]
    a[0][::5] = 0.0
    special = np.array([0.0, 5e-324, 1e-310, 2.0**-700, 2.0**-900, 1.0, 2.0**200, 2.0**-200, 2.0**201, 1e300, np.inf, np.nan])
    a[1][: m // 8] = r.choice(special, m // 8)
    u[1][m // 16: m // 4] = r.choice(special, m // 4 - m // 16)
    return np.concatenate(a), np.concatenate(u)


def _middles(m, seed):
    """a = u (q + ulp / 2), rounded: quotients next to the middle of two neighbours."""
    r = np.random.RandomState(seed)
    u, q = (np.ldexp(1.0 + r.randint(0, 1 << 52, m, dtype=np.int64) / 2.0**52, r.randint(-20, 20, m)) for _ in range(2))
    return u * q + u * np.spacing(q) * 0.5, u


def _check(f, m):
    f.argtypes = [ctypes.c_long] + [ctypes.c_void_p] * 4

    def both(a, u):
        q, p = np.empty_like(a), np.empty_like(a)
        assert f(len(a), *(x.ctypes.data for x in (a, u, q, p))) == 0
        return q, p
    a, u = _random(m, 1)
    q, p = both(a, u)
    same = (q.view(np.int64) == p.view(np.int64)) | (np.isnan(q) & np.isnan(p))
    bad = np.flatnonzero(~same)
    assert len(bad) == 0, [(float(a[i]).hex(), float(u[i]).hex(), float(q[i]).hex(), float(p[i]).hex()) for i in bad[:5]]
    q, p = both(*_middles(m, 2))
    assert np.abs(q.view(np.int64) - p.view(np.int64)).max() <= 1


def test_grouped_quotients_on_the_host(tmp_path):
    src, so = tmp_path / "div4.cpp", tmp_path / "div4.so"
    src.write_text(HOST + 'extern "C" int grouped(long n, const double *a, const double *u, double *q, double *plain)\n{\n'
                   "    for (long i = 0; i < n; i += 4) {\n" + BODY + "    }\n    return 0;\n}\n")
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, str(src), "-o", str(so)], check=True)
    _check(ctypes.CDLL(str(so)).grouped, 1 << 18)


@pytest.mark.gpu
def test_grouped_quotients_on_the_gpu(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, so = tmp_path / "div4.cu", tmp_path / "div4.so"
    src.write_text(DEVICE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-Xcompiler", "-fPIC", "-shared", "-I", CSRC, str(src), "-o",
                    str(so)], check=True)
    _check(ctypes.CDLL(str(so)).grouped, 1 << 21)

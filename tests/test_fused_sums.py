"""With multiply-adds contracted, as the fast kernels are built, the wide solver's RHS and Jacobian
sums round as the shared fragments' do: bit for bit, compiled for the CPU with fma()."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
from conftest import PKG
from radm2b200 import inputs

sys.path.insert(0, os.path.join(PKG, "mech"))
import emit  # noqa: E402
import emit_wide  # noqa: E402

SOURCE = '''
#include <cmath>
#include "radm2_wide_map.h"
#define FMAC(c, a, b) c = std::fma(a, b, c)
#define FNMA(c, a, b) c = std::fma(-(a), b, c)
#define FIX(k) fix[k]
extern "C" void general(const double *v, const double *rc, const double *fix, double ghinv, double *f, double *g)
{
#define V(i) v[i]
#define RC(r) rc[r]
#define VDOT_OUT(i, e) f[i] = (e)
#define JAC_OUT(s, e) g[s] = -(e)
#define JAC_OUT_DIAG(s, e) g[s] = (-(e)) + ghinv
#define JAC_OUT_ZERO(s, d) g[s] = (d) ? (-0.0) + ghinv : -0.0
    {
#include "radm2_fun.inc"
    }
    {
#include "radm2_jac.inc"
    }
#undef V
#undef RC
}
extern "C" void wide(double *S, const double *fix, double ghinv, double *x, double *Gm, double *Tm)
{
#define V(i) S[i]
#define RC(k) S[59 + (k)]
#define SL(k) S[k]
#define X(i) x[i]
#define GST(w, v) Gm[w] = (v)
#define TST1(c, v) Tm[(c) / 2] = (v)
#define TST_WAIT
    {
#include "radm2_wide_fun.inc"
    }
    {
#include "radm2_wide_jac.inc"
    }
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fused")
    src, so = d / "fused.cpp", d / "fused.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", os.path.join(PKG, "csrc", "gen"), str(src),
                    "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("workload,h", [("plain", 6.0), ("mixed", 600.0)])
def test_wide_sums_round_as_the_shared_ones(lib, workload, h):
    w = emit_wide.Wide(emit.load())
    cells = inputs.make_cells(32, 11, workload, 0.4)
    rc = oracle.rconst(cells["JV"], cells["TEMP"], cells["FIX"], cells["RC_N2O5"])
    ghinv = ctypes.c_double(1.0 / (h * 0.43586652150845899941601945119356))
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    fills = np.array([w.fill(s) for s in range(659)])
    for c in range(32):
        v, k, fix = (np.ascontiguousarray(a[c]) for a in (cells["VAR"], rc, cells["FIX"]))
        f, g, x = np.empty(59), np.empty(659), np.empty(59)
        lib.general(p(v), p(k), p(fix), ghinv, p(f), p(g))
        s, gm, tm = np.zeros(w.smem_words), np.zeros(w.nglobal), np.zeros(256)
        s[:59], s[59:59 + len(w.rc_rep)] = v, k[w.rc_rep]
        lib.wide(p(s), p(fix), ghinv, p(x), p(gm), p(tm))
        slots = np.array([(s, gm, tm)["SGT".index(w.kind[i])][w.pos[i] // (2 if w.kind[i] == "T" else 1)] for i in range(659)])
        assert np.array_equal(x, f)
        assert np.array_equal(slots[~fills], g[~fills])
        assert not np.array_equal(f, oracle.fun(v, fix, k))  # the contracted sums are not the plain ones

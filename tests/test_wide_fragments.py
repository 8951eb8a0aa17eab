"""The wide tensor-memory solver's generated phases (csrc/gen/radm2_wide_*.inc), compiled for
the CPU and run against the oracle.

The storage macros become arrays with the timing that the GPU allows at worst: a global load
takes its word's value where it is issued, tensor-memory loads deliver only at TLD_WAIT and
stores only at TST_WAIT (a load of a column with a store under way is an error), and slots that
the Jacobian leaves to the elimination start as NaN.  Without multiply-add contraction the
division forms equal the oracle's RHS, Jacobian, factorisation and solve bit for bit, and the
reciprocal forms the plain reciprocal fragments.
"""
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

GEN = os.path.join(PKG, "csrc", "gen")
WIDTHS = (1, 2, 4, 8, 16)


def harness():
    lines = ['''#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>
#include "radm2_wide_map.h"
static double S[RADM2_WIDE_SMEM_WORDS], Gm[RADM2_WIDE_GLOBAL_WORDS_DIV], Tm[256], x[59];
static bool under_way[256];
static int errors;
struct Load { unsigned *l, *h; double v; };
struct Store { int c; double v; };
static std::vector<Load> loads;
static std::vector<Store> stores;
static void tld(int c, unsigned &l, unsigned &h)
{
    if (c < 0 || c > 510 || c % 2 || under_way[c / 2]) errors++;
    l = h = 0xffffffffu;
    loads.push_back({&l, &h, Tm[c / 2]});
}
static void tst(int c, double v)
{
    if (c < 0 || c > 510 || c % 2) errors++;
    under_way[c / 2] = true;
    stores.push_back({c, v});
}
#define TLD_WAIT do { for (auto &q : loads) { uint64_t u; std::memcpy(&u, &q.v, 8); *q.l = (unsigned)u; *q.h = (unsigned)(u >> 32); } loads.clear(); } while (0)
#define TST_WAIT do { for (auto &q : stores) { Tm[q.c / 2] = q.v; under_way[q.c / 2] = false; } stores.clear(); } while (0)
#define TLD_GET(v) do { uint64_t u_ = ((uint64_t)v##_h << 32) | v##_l; std::memcpy(&v, &u_, 8); } while (0)
#define SL(k) S[k]
#define V(i) S[i]
#define RC(k) S[59 + (k)]
#define FIX(k) fix[k]
#define X(i) x[i]
#define GLD(v, w) v = Gm[w]
#define GST(w, v) Gm[w] = (v)
#define LU_PIVOT_CHECK(v) sing |= (v) == 0.0
#define RCPR(u) (1.0 / (u))
#define DIVR(a, u, r) ((u) == (u) && (r) != 1.0 / (u) ? (errors++, 0.0) : (a) / (u))
#define FNMA(c, a, b) c = c - (a) * (b)
#define FMAC(c, a, b) c = c + (a) * (b)
''']
    for w in WIDTHS:
        v = ["v%d" % i for i in range(w)]
        lines.append("#define TLD%d(c, %s) do { if ((c) %% %d) errors++; %s } while (0)\n"
                     % (w, ", ".join(v), 2 * w, " ".join("tld((c) + %d, %s##_l, %s##_h);" % (2 * i, a, a) for i, a in enumerate(v))))
        lines.append("#define TST%d(c, %s) do { if ((c) %% %d) errors++; %s } while (0)\n"
                     % (w, ", ".join(v), 2 * w, " ".join("tst((c) + %d, %s);" % (2 * i, a) for i, a in enumerate(v))))
    lines.append('''
extern "C" {
double *words(int which) { return which == 0 ? S : which == 1 ? Gm : which == 2 ? Tm : x; }
int fun(const double *fix) {
#include "radm2_wide_fun.inc"
    return errors; }
int jac(const double *fix, double ghinv) {
#include "radm2_wide_jac.inc"
    return errors; }
''')
    for form in ("", "_rcp"):
        lines.append('''int lu%s(int *zero) { bool sing = false;
    for (int k = 0; k < RADM2_WIDE_SPIVOTS; k++) { double &v = S[RADM2_WIDE_SPIVOT + k]; LU_PIVOT_CHECK(v); %s }
#include "radm2_wide_lu%s.inc"
    *zero = sing; return errors; }
int solve%s() {
#include "radm2_wide_solve%s.inc"
    return errors; }
''' % (form, "v = 1.0 / v;" if form else "Gm[RADM2_WIDE_GRCP + k] = 1.0 / v;", form, form, form))
    # the plain reciprocal fragments on an array of slots, for the reciprocal forms
    lines.append('''
#undef LU_PIVOT_CHECK
#define LU_PIVOT_CHECK(k, v) (void)0
#define LU_T double
#define G(s) g[s]
void plain_rcp(double *g, double *x) {
#include "radm2_decomp_rcp.inc"
#include "radm2_solve_rcp.inc"
}
''')
    return "".join(lines) + "}\n"


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("wide")
    src, so = d / "wide.cpp", d / "wide.so"
    src.write_text(harness())
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", GEN, str(src), "-o", str(so)],
                   check=True)
    h = ctypes.CDLL(str(so))
    h.words.restype = ctypes.POINTER(ctypes.c_double)
    h.jac.argtypes = [ctypes.c_void_p, ctypes.c_double]
    h.fun.argtypes = [ctypes.c_void_p]
    h.plain_rcp.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    return h


@pytest.fixture(scope="module")
def wide():
    return emit_wide.Wide(emit.load())


class Words:
    def __init__(self, lib, wide):
        size = {0: wide.smem_words, 1: wide.nglobal + 59, 2: 256, 3: 59}
        self.s, self.g, self.t, self.x = (np.ctypeslib.as_array(lib.words(i), (size[i],)) for i in range(4))
        self.wide = wide

    def slot(self, s):
        k, p = self.wide.kind[s], self.wide.pos[s]
        return (self.s, p) if k == "S" else (self.g, p) if k == "G" else (self.t, p // 2)

    def slots(self):
        return np.array([a[i] for a, i in map(self.slot, range(659))])


def test_every_slot_has_a_word_of_its_own(wide):
    seen = {(wide.kind[s], wide.pos[s]) for s in range(659)}
    assert len(seen) == 659
    assert sorted(p for k, p in seen if k == "T") == list(range(0, 512, 2))
    assert {p for k, p in seen if k == "S"} == set(range(59 + len(wide.rc_rep), wide.smem_words))
    assert {p for k, p in seen if k == "G"} == set(range(emit_wide.GLU, wide.nglobal))
    assert (wide.smem_words * 1024 + 64) <= 227 * 1024


def test_committed_fragments_are_the_emitter_s(wide, tmp_path, monkeypatch):
    monkeypatch.setattr(emit_wide, "CSRC_GEN", str(tmp_path))
    emit_wide.main()
    for name in os.listdir(tmp_path):
        assert (tmp_path / name).read_text() == open(os.path.join(GEN, name)).read(), name


def test_repeated_rate_constants_share_a_word(wide):
    cells = inputs.make_cells(64, 5, "mixed", 0.4)
    rc = oracle.rconst(cells["JV"], cells["TEMP"], cells["FIX"], cells["RC_N2O5"])
    for r, w in enumerate(wide.rc_word):
        want = float(wide.m["rconst"][r][1]) if w is None else rc[:, wide.rc_rep[w]]
        assert np.array_equal(rc[:, r], np.broadcast_to(want, 64))


@pytest.mark.parametrize("workload,h", [("plain", 6.0), ("mixed", 1.0e-3), ("mixed", 600.0)])
def test_phases_equal_the_oracle(lib, wide, workload, h):
    cells = inputs.make_cells(16, 11, workload, 0.4)
    rc = oracle.rconst(cells["JV"], cells["TEMP"], cells["FIX"], cells["RC_N2O5"])
    per_cell = lambda f: np.array([f(cells["VAR"][c], cells["FIX"][c], rc[c]) for c in range(16)])  # noqa: E731
    f_o, j_o = per_cell(oracle.fun), per_cell(oracle.jac)
    ghinv = 1.0 / (h * 0.43586652150845899941601945119356)
    w = Words(lib, wide)
    fills = [s for s in range(659) if wide.fill(s)]
    for c in range(16):
        fix = np.ascontiguousarray(cells["FIX"][c])
        w.s[:59] = cells["VAR"][c]
        w.s[59:59 + len(wide.rc_rep)] = rc[c][wide.rc_rep]
        assert lib.fun(fix.ctypes.data) == 0
        assert np.array_equal(w.x, f_o[c])
        g = -j_o[c]
        g[wide.diag] += ghinv
        zero = ctypes.c_int()
        for form in ("", "_rcp"):
            for s in range(659):
                a, i = w.slot(s)
                a[i] = np.nan
            assert lib.jac(fix.ctypes.data, ghinv) == 0
            stored = np.setdiff1d(np.arange(659), fills)
            assert np.array_equal(w.slots()[stored], g[stored]) and not g[fills].any()
            assert getattr(lib, "lu" + form)(ctypes.byref(zero)) == 0 and zero.value == 0
            if form:
                lu_o, x_o = g.copy(), f_o[c].copy()
                lib.plain_rcp(lu_o.ctypes.data, x_o.ctypes.data)
            else:
                lu_o, _ = oracle.decomp(g)
                x_o = oracle.solve(lu_o, f_o[c])
            assert np.array_equal(w.slots(), lu_o)
            w.x[:] = f_o[c]
            assert getattr(lib, "solve" + form)() == 0
            assert np.array_equal(w.x, x_o)


def test_zero_pivot_is_seen(lib, wide):
    w = Words(lib, wide)
    zero = ctypes.c_int()
    for row in (0, 18, 58):
        for s in range(659):
            a, i = w.slot(s)
            a[i] = 1.0 if s in wide.diag else 0.0
        a, i = w.slot(wide.diag[row])
        a[i] = 0.0
        assert lib.lu(ctypes.byref(zero)) == 0 and zero.value == 1

"""The wide tensor-memory solver (csrc/radm2_wide.cuh) on the routes that lead to it: the
library's own launch shape (block_threads 0) of either schedule, the explicit wide placement,
and the general kernels for rate constants set by the caller.

SAME_ARITH for kernels that compile the same expressions; 1e-10 and equal step counts against
the oracle, as for every FP64 kernel.
"""
import numpy as np
import pytest

import oracle
import radm2b200
from conftest import ATOL, RTOL, SAME_ARITH, rel_err
from radm2b200 import inputs

pytestmark = pytest.mark.gpu
STATIC, PERS = radm2b200.SCHED_STATIC, radm2b200.SCHED_PERSISTENT
WIDE = radm2b200.lib.PLACE_LU_TMEM_WIDE


def run(cells, order=None, rc=None, **opts):
    with radm2b200.Solver(**opts) as s:
        s.set_cells(cells)
        s.update_rconst()
        if rc is not None:
            s.set_rconst(rc)
        if order is not None:
            s.set_cell_order(order)
        got = s.get_rconst()
        ipar, rpar = radm2b200.default_params(hstart=6.0)
        ierr = s.rosenbrock(0.0, 600.0, ATOL, RTOL, rpar, ipar)
        assert ierr == 1
        return s.get_state(), s.cell_stats(), got


# one lane, a warp's edge, a block's edges, more cells than lanes of one block, more blocks than SMs
@pytest.mark.parametrize("parity", [0, 1])
@pytest.mark.parametrize("n", [1, 32, 127, 128, 129, 1000, 20000])
def test_library_shape_matches_oracle(n, parity):
    cells = inputs.make_cells(n, 31, "plain", 0.3)
    y, st, rc = run(cells, parity=parity)
    yp, stp, _ = run(cells, schedule=PERS, parity=parity)
    yw, stw, _ = run(cells, schedule=PERS, placement=WIDE, parity=parity)
    assert np.array_equal(y, yp) and np.array_equal(y, yw)  # one kernel: when a cell is taken does not matter
    assert all(np.array_equal(st[k], q[k]) for q in (stp, stw) for k in st)
    pick = np.arange(n) if n <= 1000 else np.arange(0, n, 23)
    ipar, rpar = radm2b200.default_params(hstart=6.0)
    _, p = oracle.params(0.0, 600.0, ATOL, RTOL, rpar, ipar)
    y_o, st_o = oracle.integrate(cells["VAR"][pick], cells["FIX"][pick], rc[pick], p)
    assert np.array_equal(st["nacc"][pick], st_o["nacc"]) and np.array_equal(st["nrej"][pick], st_o["nrej"])
    assert rel_err(y[pick], y_o).max() <= 1e-10


def test_visiting_order_does_not_matter():
    cells = inputs.make_cells(3001, 7, "mixed", 0.4)
    order = np.random.RandomState(1).permutation(3001).astype(np.int32)
    y, st, _ = run(cells, schedule=PERS)
    for schedule in (STATIC, PERS):
        yo, sto, _ = run(cells, order=order, schedule=schedule)
        assert np.array_equal(y, yo) and np.array_equal(st["nacc"], sto["nacc"])


@pytest.mark.parametrize("opts", [dict(schedule=STATIC), dict(schedule=PERS), dict(schedule=PERS, placement=WIDE)])
def test_rate_constants_set_by_the_caller(opts):
    """Constants that no formula gives (every one of the 156 its own): the general kernels, within
    SAME_ARITH of the explicit 128-thread launch, and the formulas again after update_rconst."""
    cells = inputs.make_cells(700, 3, "plain", 0.3)
    y0, st0, rc = run(cells, **opts)
    own = rc * (1.0 + 1.0e-3 * np.arange(156) / 156.0)
    y, st, got = run(cells, rc=own, **opts)
    assert np.array_equal(got, own)
    y1, st1, _ = run(cells, rc=own, schedule=PERS, block_threads=128)
    assert np.array_equal(st["nacc"], st1["nacc"]) and rel_err(y, y1).max() <= SAME_ARITH
    assert rel_err(y, y0).max() > 1e-6
    with radm2b200.Solver(**opts) as s:
        s.set_cells(cells)
        s.set_rconst(own)
        s.update_rconst()
        ipar, rpar = radm2b200.default_params(hstart=6.0)
        assert s.rosenbrock(0.0, 600.0, ATOL, RTOL, rpar, ipar) == 1
        assert np.array_equal(s.get_state(), y0)


@pytest.mark.parametrize("atol", [1.0e-160, 1.0, 1.0e160])
def test_error_norm_beyond_the_branch_free_range(atol):
    """Tolerances whose squares leave div_newton's range take the plain division: the norms, and so
    the step counts, are those of the global-scratch kernel.  (At 1e160 nothing limits the steps
    and the states amplify any rounding, so only the counts are compared there.)"""
    cells = inputs.make_cells(200, 13, "plain", 0.3)
    out = []
    for block in (0, 128):
        with radm2b200.Solver(schedule=PERS, block_threads=block) as s:
            s.set_cells(cells)
            ipar, rpar = radm2b200.default_params(hstart=6.0, max_steps=400)
            ierr = s.rosenbrock(0.0, 600.0, np.full(59, atol), RTOL, rpar, ipar)
            out.append((ierr, s.get_state(), s.cell_stats()))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][2]["nacc"], out[1][2]["nacc"]) and np.array_equal(out[0][2]["status"], out[1][2]["status"])
    assert np.array_equal(out[0][2]["nrej"], out[1][2]["nrej"])
    if atol < 1.0e100:
        assert rel_err(out[0][1], out[1][1]).max() <= SAME_ARITH


@pytest.mark.parametrize("h", [1.0e-40, 1.0e-6, 600.0, 1.0e40])
def test_pivot_divisions_over_the_exponent_range(h):
    """Reference arithmetic divides by a pivot through its reciprocal; steps that put the pivots
    1 / (h gamma) outside 2^-100 .. 2^100 (and zero multipliers, at night) take the plain division.
    Bit for bit the global-scratch kernel of the same arithmetic."""
    cells = inputs.make_cells(130, 17, "mixed", 0.5)
    out = []
    for block in (0, 128):
        with radm2b200.Solver(parity=1, block_threads=block) as s:
            s.set_cells(cells)
            ipar, rpar = radm2b200.default_params(hstart=h, max_steps=6)
            rpar[0] = min(h, 1.0e-30)
            ierr = s.rosenbrock(0.0, max(h, 600.0), ATOL, RTOL, rpar, ipar)
            out.append((ierr, s.get_state(), s.cell_stats()))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1], equal_nan=True)
    assert all(np.array_equal(out[0][2][k], out[1][2][k], equal_nan=True) for k in out[0][2])


@pytest.mark.parametrize("nchunk", [2, 3, 8, 17])
def test_chunks_on_two_streams(nchunk):
    """Odd chunks run on a second stream with their own scratch, seeded from their own rows of the
    network's work arrays: bit for bit one chunk's result, call after call."""
    from radm2b200 import seeding
    cells = inputs.make_cells(20011, 5, "mixed", 0.4)
    net = seeding.load_net(seeding.DEFAULT_NET)
    with radm2b200.Solver(schedule=PERS, placement=WIDE) as s:
        s.set_cells(cells)
        s.attach_mlp(net)
        out = []
        for k in (1, nchunk, nchunk):
            y = np.ascontiguousarray(cells["VAR"]).copy()
            ipar, rpar = radm2b200.default_params(hstart=6.0)
            assert s.rosenbrock_host(y, cells["FIX"], cells["TEMP"], cells["RC_N2O5"], cells["JV"], 0.0, 600.0, ATOL, RTOL, rpar,
                                     ipar, nchunk=k) == 1
            out.append((y, list(ipar[10:17])))
        s.attach_mlp(None)
    assert all(np.array_equal(y, out[0][0]) and c == out[0][1] for y, c in out[1:])

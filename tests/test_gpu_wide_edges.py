"""Contexts that leave the launch shape to the library (the wide solver) at its edges -- step cap,
non-finite cells, warps with idle lanes, error norms of zeros -- against the explicit
global-scratch kernels, and those kernels, schedule by schedule, against the oracle."""
import numpy as np
import pytest

import oracle
import radm2b200
from conftest import ATOL, RTOL, SAME_ARITH, rel_err
from radm2b200 import inputs

pytestmark = pytest.mark.gpu
STATIC, PERS = radm2b200.SCHED_STATIC, radm2b200.SCHED_PERSISTENT
PARITY = 1e-10


def run(cells, atol=ATOL, max_steps=0, **opts):
    with radm2b200.Solver(**opts) as s:
        s.set_cells(cells)
        s.update_rconst()
        rc = s.get_rconst()
        ipar, rpar = radm2b200.default_params(hstart=6.0, max_steps=max_steps)
        ierr = s.rosenbrock(0.0, 600.0, atol, RTOL, rpar, ipar)
        return ierr, s.get_state(), s.cell_stats(), rc, list(ipar[10:17])


@pytest.mark.parametrize("block", [64, 128])
@pytest.mark.parametrize("n", [1, 65, 1000])
def test_explicit_shapes_of_both_schedules_match_the_oracle(n, block):
    cells = inputs.make_cells(n, 37, "plain", 0.3)
    ipar, rpar = radm2b200.default_params(hstart=6.0)
    _, p = oracle.params(0.0, 600.0, ATOL, RTOL, rpar, ipar)
    ys = []
    for schedule in (STATIC, PERS):
        ierr, y, st, rc, _ = run(cells, schedule=schedule, block_threads=block)
        y_o, st_o = oracle.integrate(cells["VAR"], cells["FIX"], rc, p)
        assert ierr == 1
        assert np.array_equal(st["nacc"], st_o["nacc"]) and np.array_equal(st["nrej"], st_o["nrej"])
        assert rel_err(y, y_o).max() <= PARITY
        ys.append(y)
    assert rel_err(ys[1], ys[0]).max() <= SAME_ARITH


@pytest.mark.parametrize("schedule", [STATIC, PERS])
@pytest.mark.parametrize("parity", [0, 1])
def test_step_cap_and_nonfinite_cells(schedule, parity):
    """The same outcome per cell as on the global-scratch kernel (bit for bit in reference
    arithmetic), whatever the neighbours in the warp do."""
    cells = inputs.make_cells(300, 3, "mixed", 0.4)
    cells["VAR"][5, 45] = np.nan
    cells["VAR"][130, 3] = np.inf
    cells["VAR"][200] = 0.0
    for cap in (5, 300):
        out = [run(cells, max_steps=cap, schedule=schedule, parity=parity, block_threads=b) for b in (0, 128)]
        (ierr, y, st, _, counters), (ierr0, y0, st0, _, counters0) = out
        assert ierr == ierr0 < 0
        assert all(np.array_equal(st[k], st0[k]) for k in ("status", "nacc", "nrej")) and counters == counters0
        assert st["status"][5] < 0 and (cap > 5 or (st["status"][:5] == -6).all())
        fin = np.isfinite(y0).all(axis=1)
        assert np.array_equal(y[~fin], y0[~fin], equal_nan=True) and fin.sum() >= 298
        if parity:
            assert np.array_equal(y[fin], y0[fin]) and np.array_equal(np.signbit(y[fin]), np.signbit(y0[fin]))
        else:
            assert rel_err(y[fin], y0[fin]).max() <= SAME_ARITH


@pytest.mark.parametrize("atol", [1.0e-170, 1.0e-152, 1.0e-75, 1.0])
@pytest.mark.parametrize("n", [1, 33])
def test_error_norm_of_zeros(n, atol):
    """Species that stay zero have a zero error; with a tolerance whose square vanishes the norm is
    0 / 0, as the plain division gives it.  Idle lanes have nothing but zeros."""
    cells = inputs.make_cells(n, 41, "plain", 0.3)
    cells["VAR"][:, ::7] = 0.0
    cells["VAR"][n // 2] = 0.0
    out = [run(cells, atol=np.full(59, atol), max_steps=60, parity=1, block_threads=b) for b in (0, 128)]
    assert out[0][0] == out[1][0]
    assert all(np.array_equal(out[0][2][k], out[1][2][k], equal_nan=True) for k in out[0][2])
    assert np.array_equal(out[0][1], out[1][1], equal_nan=True)

"""Contexts that leave the launch shape to the library (the wide solver) at its edges, against the
explicit global-scratch kernels."""
import numpy as np
import pytest

import radm2b200
from conftest import ATOL, RTOL
from radm2b200 import inputs

pytestmark = pytest.mark.gpu


def run(cells, atol=ATOL, max_steps=0, **opts):
    with radm2b200.Solver(**opts) as s:
        s.set_cells(cells)
        s.update_rconst()
        rc = s.get_rconst()
        ipar, rpar = radm2b200.default_params(hstart=6.0, max_steps=max_steps)
        ierr = s.rosenbrock(0.0, 600.0, atol, RTOL, rpar, ipar)
        return ierr, s.get_state(), s.cell_stats(), rc, list(ipar[10:17])


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

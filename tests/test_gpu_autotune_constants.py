"""The autotuner times the kernels that the context will run: with rate constants set by the caller,
on those constants."""
import numpy as np
import pytest

import radm2b200
from conftest import ATOL, RTOL
from radm2b200 import inputs

pytestmark = pytest.mark.gpu


def attempts(s):
    ipar, rpar = radm2b200.default_params()
    assert s.run_split(1, 600.0, ATOL, RTOL, rpar, ipar) == 1
    return int(ipar[13]) + int(ipar[14])


@pytest.mark.parametrize("n,sample", [(2048, 0), (4100, 1025)])
def test_sample_takes_the_caller_s_constants(n, sample):
    cells = inputs.make_cells(n, 12, "mixed", 0.4)
    with radm2b200.Solver() as s:
        s.set_cells(cells)
        rc = s.get_rconst()
        formula = {t["attempts"] for t in s.autotune(600.0, ATOL, RTOL, sample_cells=sample) if t["ms"] > 0}
    own = rc * np.linspace(0.2, 3.0, 156)
    pick = np.arange(0, n, n // (sample or n))[:sample or n]
    with radm2b200.Solver() as s:
        s.set_cells({k: np.ascontiguousarray(v[pick]) for k, v in cells.items() if k != "cls"})
        s.set_rconst(np.ascontiguousarray(own[pick]))
        want = attempts(s)
    with radm2b200.Solver() as s:
        s.set_cells(cells)
        s.set_rconst(own)
        got = {t["attempts"] for t in s.autotune(600.0, ATOL, RTOL, sample_cells=sample) if t["ms"] > 0}
        assert got == {want} and formula != got
        assert np.array_equal(s.get_rconst(), own)
        s.set_cells(cells)  # the formulas' constants again, for the sample as well
        assert {t["attempts"] for t in s.autotune(600.0, ATOL, RTOL, sample_cells=sample) if t["ms"] > 0} == formula

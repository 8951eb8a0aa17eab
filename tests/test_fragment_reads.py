"""The shared RHS and Jacobian fragments read a product's factors once.  A use that names V(i) or
RC(r) again costs a second load in the kernels whose working set lies in memory: a store in between
might have changed them for all the compiler knows."""
import os
import re

import pytest

from conftest import PKG


@pytest.mark.parametrize("name", ["radm2_fun.inc", "radm2_jac.inc"])
def test_sums_read_factors_from_locals(name):
    text = open(os.path.join(PKG, "csrc", "gen", name)).read()
    sums = re.findall(r"F(?:MAC|NMA)\(.*\);", text)
    assert len(sums) > 100
    assert [s for s in sums if re.search(r"\b(V|RC|FIX)\(", s)] == []

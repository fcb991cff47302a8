"""A basis far larger than the solve comes to use (ncv 7390 of 7400 unknowns; the pair
converges within the first tens of vectors), and the solves after it on the same
context: nothing depends on the size of the largest basis so far but the buffers."""
import numpy as np
import pytest

from tailor_gb300 import api
from tailor_gb300.case import Physics, make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [1, 0])
def test_large_basis_and_after(gpu_lib, precision):
    ph = Physics(alpha=1.4, reynolds=700.0, nev=1, tol=1e-9)
    with api.Problem(make_case(40, 37, physics=ph)) as p:
        api.run_pipeline(p)
        kw = dict(nev=1, precision=precision, fallback=False)
        large = api.EigenSolver(p).solve(ncv=7390, **kw)
        after = api.EigenSolver(p).solve(ncv=60, **kw)
    assert large.diag["iterations"] == 1
    for s in (large, after):
        assert len(s.lam) == 1 and s.residual[0] <= 1e-9
    assert abs(large.lam[0] - after.lam[0]) <= 1e-7 * abs(after.lam[0])

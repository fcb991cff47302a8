"""The mixed form's pipelined operator applications (three right-hand sides
per triangular solve) against the FP64 form with the same basis size: sizes that leave remainders in
the node-wise kernels (51 nodes per CTA) and block rows (8 per CTA), bases
down to three vectors (a restart after every second application), real and complex
targets, and both solve-block sizes.  Every application is accepted at
||B v - K x|| <= 1e-12 ||B v||, so eigenvalues of eigen residual <= 1e-10
agree to the parity bar of 1e-8."""
import numpy as np
import pytest

from tailor_gb300 import api
from tailor_gb300.case import Physics, make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nz,nev,ncv,omega,solve_block", [
    (24, 16, 4, 0, 0j, 0),            # 384 nodes: 7 whole CTAs and 27 nodes
    (17, 12, 1, 3, 0j, 0),            # 204 = 4 x 51 nodes; a basis of three
    (31, 18, 3, 5, 0.3 + 0.01j, 128),  # odd rows, complex target
    (60, 32, 8, 40, 0.1 + 0j, 0),     # several diagonal blocks per front
])
def test_matches_the_fp64_form(gpu_lib, ny, nz, nev, ncv, omega, solve_block):
    ph = Physics(alpha=1.4, reynolds=700.0, omega=omega, nev=nev, tol=1e-10, max_it=3000)
    with api.Problem(make_case(ny, nz, physics=ph)) as p:
        api.run_pipeline(p)
        ref = api.EigenSolver(p).solve(nev=nev, ncv=ncv, precision=0)
        sol = api.EigenSolver(p).solve(nev=nev, ncv=ncv, precision=1, solve_block=solve_block,
                                       fallback=False)
    assert len(sol.lam) == nev and np.all(sol.residual <= 1e-10)
    assert 0.0 < sol.diag["refine_res"][2] <= 1e-12
    # three vectors per triangular solve, one correction of x in each
    assert sol.diag["solves"] == 3 * sol.diag["trisolves"]
    for lam in sol.lam:
        assert np.min(np.abs(ref.lam - lam)) <= 1e-8 * abs(lam)

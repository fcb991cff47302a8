"""The pipelined applications at grids that leave every kind of remainder in their
kernels (10 nodes per CTA in the start and the shift, 12 in the targets, 16 block rows
per CTA in the residuals), and on operators that a round does not contract, where the
single application takes over and the guesses go on from its result: eigenvalues of
eigen residual <= 1e-10 against the FP64 form with the same basis."""
import numpy as np
import pytest

from tailor_gb300 import api
from tailor_gb300.case import Physics, make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nz,left", [
    (17, 17, (9, 1, 1)),    # 289 nodes: remainders modulo 10, 12 and 16
    (23, 13, (9, 11, 11)),  # 299
    (17, 15, (5, 3, 15)),   # 255
    (17, 13, (1, 5, 13)),   # 221
])
def test_remainders(gpu_lib, ny, nz, left):
    assert tuple(ny * nz % k for k in (10, 12, 16)) == left
    ph = Physics(alpha=1.4, reynolds=700.0, nev=3, tol=1e-10, max_it=3000)
    with api.Problem(make_case(ny, nz, physics=ph)) as p:
        api.run_pipeline(p)
        ref = api.EigenSolver(p).solve(nev=3, ncv=20, precision=0)
        sol = api.EigenSolver(p).solve(nev=3, ncv=20, precision=1, fallback=False)
    assert len(sol.lam) == 3 and np.all(sol.residual <= 1e-10)
    for lam in sol.lam:
        assert np.min(np.abs(ref.lam - lam)) <= 1e-8 * abs(lam)


@pytest.mark.parametrize("distance", [1e-2, 1e-3, 1e-4])
def test_a_round_that_does_not_contract(gpu_lib, distance):
    """sigma at a small distance from an eigenvalue: cond(K) of 1e4 to 1e6 and a
    complex64 factor that contracts too little.  Only the single application's loop
    ends above 1e-12 (it stops at the rounding floor), so the largest accepted residual
    says that it ran."""
    n = 303
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(2 * n)
    ref = np.linalg.eigvals(A)
    near = ref[np.argmin(np.abs(ref - (0.3 - 0.2j)))]
    kw = dict(omega=complex(-near.imag, near.real), sigma=near * (1 + distance), nev=3,
              modes=False, max_it=60)
    sol = api.solve_pencil(A, np.eye(n, dtype=complex), precision=1, fallback=False, **kw)
    plain = api.solve_pencil(A, np.eye(n, dtype=complex), precision=0, **kw)
    assert np.all(sol.residual <= 1e-10) and len(sol.lam) == 3
    for lam in sol.lam:
        assert np.min(np.abs(plain.lam - lam)) <= 1e-8 * abs(lam)
    if distance <= 1e-4:
        assert sol.diag["refine_res"][2] > 1e-12

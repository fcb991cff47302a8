"""The complex64 factor in inverse form (one product per front and
direction) against the block-step solves, through tlr_factor_solve: pivot
blocks of one, several and many 256-row diagonal blocks with remainders, a
single dense front (a pencil), split and unsplit row tiles.

The block-step factor of the same matrix comes from cuda_core_schur = 1.
Both are complex64 factorisations of K; with E = K x - r their residuals
||E|| / ||r|| are bounded by growth x n x 2^-24 x cond-free constants: 1e-2
covers the explicit inverses at these sizes, and 1e-3 relative agreement of
one refinement step separates a wrong entry from rounding."""
import numpy as np
import pytest

from tailor_gb300 import api
from tailor_gb300.case import Physics, make_case

pytestmark = pytest.mark.gpu


def _solve(p, rhs, multi):
    nv, n = rhs.shape
    r = np.ascontiguousarray(np.stack([rhs.real, rhs.imag], -1))
    out = np.zeros_like(r)
    st = p.lib.tlr_factor_solve(p.ctx, nv, r.ctypes.data, out.ctypes.data, multi)
    assert st == 0, p.lib.tlr_last_error(p.ctx)
    return out[..., 0] + 1j * out[..., 1]


@pytest.mark.parametrize("ny,nz,cuda_core", [
    (24, 16, 0), (24, 16, 1),   # fronts of one diagonal block
    (60, 32, 0), (60, 32, 1),   # up to four blocks, the last one of 32 rows
    (83, 47, 0), (83, 47, 1),   # up to five blocks, odd row counts
])
def test_factor_solve_residual(gpu_lib, ny, nz, cuda_core):
    ph = Physics(alpha=1.3, omega=0j, nev=4, tol=1e-10)
    with api.Problem(make_case(ny, nz, physics=ph)) as p:
        api.run_pipeline(p)
        api.EigenSolver(p).solve(nev=4, precision=1, cuda_core_schur=cuda_core, fallback=False)
        rng = np.random.default_rng(7)
        n = 5 * p.case.nodes
        v = rng.standard_normal((4, n)) + 1j * rng.standard_normal((4, n))
        b = np.stack([p.spmv(api.TLR_MAT_B, q) for q in v])
        x = _solve(p, b, 1)
        assert np.array_equal(x, _solve(p, b, 0))
        for q in range(4):  # sigma = 0: K = A
            r = b[q] - p.spmv(api.TLR_MAT_A, x[q])
            assert np.linalg.norm(r) <= 1e-2 * np.linalg.norm(b[q])
            # a correction contracts it again
            x2 = x[q] + _solve(p, r[None], 0)[0]
            r2 = b[q] - p.spmv(api.TLR_MAT_A, x2)
            assert np.linalg.norm(r2) <= 1e-2 * np.linalg.norm(r)


@pytest.mark.parametrize("n", [10, 255, 303, 520, 1300])
def test_pencil_single_front(gpu_lib, n):
    """One dense front of order n (1 to 6 diagonal blocks): mixed-form
    eigenvalues within 1e-8 of the dense solver's."""
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(2 * n)
    B = np.eye(n, dtype=complex)
    sol = api.solve_pencil(A, B, omega=complex(0.1, 0.2), nev=2, precision=1, ncv=min(n - 1, 40),
                           fallback=False)
    z = complex(0.2, -0.1)
    ref = np.linalg.eigvals(A)
    ref = ref[np.argsort(np.abs(ref - z))][:2]
    for lam in sol.lam:
        assert np.min(np.abs(ref - lam)) <= 1e-8 * max(abs(lam), 0.1)

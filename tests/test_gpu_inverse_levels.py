"""Inverse-form solves over levels of both kinds -- those whose forward items
collect the right-hand side and the children themselves (at most 131072 columns
of 32 rows) and those with a gather launch -- through tlr_factor_solve: a tree of
small levels only (24 x 16, 60 x 32) and one with large levels below small ones
(100 x 50, 518 MB of factor).  The residual bound is that of the complex64
factor; several vectors at once must give the bits of one at a time."""
import numpy as np
import pytest

from tailor_gb300 import api
from tailor_gb300.case import Physics, make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nz", [(24, 16), (60, 32), (100, 50)])
def test_small_and_large_levels(gpu_lib, ny, nz):
    ph = Physics(alpha=1.3, omega=0j, nev=2, tol=1e-10)
    with api.Problem(make_case(ny, nz, physics=ph)) as p:
        api.run_pipeline(p)
        api.EigenSolver(p).solve(nev=2, precision=1, fallback=False)
        rng = np.random.default_rng(11)
        n = 5 * p.case.nodes
        v = rng.standard_normal((4, n)) + 1j * rng.standard_normal((4, n))
        b = np.stack([p.spmv(api.TLR_MAT_B, q) for q in v])
        rhs = np.ascontiguousarray(np.stack([b.real, b.imag], -1))
        got = []
        for multi in (0, 1):
            out = np.zeros_like(rhs)
            assert p.lib.tlr_factor_solve(p.ctx, 4, rhs.ctypes.data, out.ctypes.data, multi) == 0
            got.append(out[..., 0] + 1j * out[..., 1])
        assert np.array_equal(got[0], got[1])
        for q in range(4):  # sigma = 0: K = A
            r = b[q] - p.spmv(api.TLR_MAT_A, got[0][q])
            assert np.linalg.norm(r) <= 1e-2 * np.linalg.norm(b[q])

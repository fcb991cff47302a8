"""The persistent Schur update of complex64 fronts (F22 tiles copied to shared
memory as 16-byte aligned ranges of columns that start on any 8-byte boundary)
against the kernel that takes one tile per CTA and reads F22 directly: the same
products in the same order, so the factors and the solves must agree bit for bit.

Grids with fronts of odd and even leading dimensions, remainders of the 128-row
and 64-column tiles, panels of 32, 64 and 128 columns."""
import numpy as np
import pytest

from tailor_gb300 import api
from tailor_gb300.case import Physics, make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nz,panel", [(24, 16, 0), (41, 23, 0), (83, 47, 32), (60, 32, 128)])
def test_persistent_update_bits(gpu_lib, ny, nz, panel):
    ph = Physics(alpha=1.3, omega=0j, nev=2, tol=1e-10)
    with api.Problem(make_case(ny, nz, physics=ph)) as p:
        api.run_pipeline(p)
        rng = np.random.default_rng(2)
        rhs = rng.standard_normal((2, 5 * p.case.nodes, 2))
        got = []
        for kernel in (0, 4):
            api.EigenSolver(p).solve(nev=2, precision=1, panel_width=panel,
                                     cuda_core_schur=kernel, fallback=False)
            out = np.zeros_like(rhs)
            assert p.lib.tlr_factor_solve(p.ctx, 2, rhs.ctypes.data, out.ctypes.data, 0) == 0
            got.append(out)
        assert np.all(np.isfinite(got[0]))
        assert np.array_equal(got[0], got[1])

"""Mixed-form solves whose operator's powers leave FP32's range: a pencil scaled by
powers of ten.  OP scales by the inverse, so the pipelined guesses of OP^2 v and OP^3 v
overflow at 1e-14 and below and vanish at 1e14 and above; the eigenvalues scale with the
pencil all the same, to the tolerance of 1e-10, and the solve takes no more triangular
solves than single applications (three each) and a few rounds of three before the
guesses are given up.  A null right-hand scale would make a case fail, so the extremes
stay ten orders inside FP32's range."""
import numpy as np
import pytest

from tailor_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [-25, -14, -9, 9, 14, 25])
def test_scaled_pencil(gpu_lib, exponent):
    n, z, s = 120, complex(0.3, -0.2), 10.0 ** exponent
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(2 * n)
    B = np.eye(n, dtype=complex)
    ref = np.linalg.eigvals(A)
    ref = ref[np.argsort(np.abs(ref - z))]
    kw = dict(nev=3, precision=1, fallback=False, modes=False, max_it=60)
    one = api.solve_pencil(A, B, omega=complex(-z.imag, z.real), **kw)
    sol = api.solve_pencil(A * s, B, omega=complex(-z.imag, z.real) * s, **kw)
    assert len(sol.lam) == 3 and np.all(sol.residual <= 1e-10)
    for lam in sol.lam:
        assert np.min(np.abs(ref[:6] * s - lam)) <= 1e-9 * abs(lam)
    # applications: the unscaled solve's rounds are at most one per application
    # more than needed, a scaled one's applications are as many or one check more
    assert sol.diag["solves"] <= one.diag["solves"] + 60

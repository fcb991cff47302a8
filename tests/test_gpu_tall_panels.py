"""Pivoting panels taller than eight CTAs' shared memory (more than 2800 fully
summed rows; one dense front of a pencil) on a cluster of 16, against the one-CTA
panel: the same pivots and arithmetic, so the eigenvalues agree to the bit."""
import numpy as np
import pytest

from tailor_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,precision", [(2803, 1), (3100, 1), (3100, 0)])
def test_sixteen_cta_panel_is_bitwise_the_single_cta_panel(gpu_lib, n, precision):
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(2 * n)
    B = np.eye(n, dtype=complex)
    lam = [api.solve_pencil(A, B, omega=complex(0.1, 0.2), nev=1, ncv=60, precision=precision,
                            cluster_panel=c, fallback=False).lam for c in (-1, 0)]
    assert np.array_equal(lam[0], lam[1])

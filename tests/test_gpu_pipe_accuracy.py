"""Pipelined applications of a well-conditioned pencil are as accurate as three
dependent solves: not merely within the acceptance limit of 1e-12, but at the rounding of
the float-float residual that refines them, two times 2^-47 cond(K) (three corrections by
a complex64 factor leave (2^-24 cond K)^3, far below)."""
import numpy as np
import pytest

from tailor_gb300 import api

pytestmark = pytest.mark.gpu


def _random(n):
    rng = np.random.default_rng(n)
    return (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(2 * n)


@pytest.mark.parametrize("A,z", [
    (_random(8), 0.3 - 0.2j), (_random(10), 0.3 - 0.2j),
    (np.diag(np.linspace(0.1, 3, 120) * (1 + 0.3j)), 0.31 + 0.02j),
], ids=["random8", "random10", "diagonal120"])
def test_residual_of_the_applications(gpu_lib, A, z):
    n = len(A)
    sol = api.solve_pencil(A, np.eye(n, dtype=complex), omega=complex(-z.imag, z.real),
                           nev=1 if n < 100 else 3, precision=1, fallback=False, modes=False)
    cond = np.linalg.cond(A - z * np.eye(n))
    assert cond < 50
    assert 0 < sol.diag["refine_res"][2] <= 2 * 2.0 ** -47 * cond

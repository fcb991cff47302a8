"""Solves through the complex128 factor by sliced products against solves through the
one by FP64 FMAs (cuda_core_schur = 1): residuals b - K x in extended precision, on
pencils whose entries span up to sixteen decades without any structure (or in blocks, by
rows, by columns), and on a grid.

A slice number holds its entry to 2^-54 of the largest entry of its line, not to 53
bits of its own, so a product of such entries alone loses more than FMAs do.  In a
factor the multipliers are at most one and a line's largest products carry the
rounding of either kind, so the backward errors have one size.  Each factorisation
draws its roundings once; two draws of one distribution lie within a factor of 3
(norms over four right-hand sides)."""
import numpy as np
import pytest

from tailor_gb300 import api
from tailor_gb300.case import Physics, make_case

pytestmark = pytest.mark.gpu


def _solve(p, cuda_core, b):
    try:  # one restart: only its factor is wanted
        api.EigenSolver(p).solve(nev=1, precision=0, cuda_core_schur=cuda_core, max_it=1)
    except api.TailorError as e:
        assert e.status == 13
    x = np.zeros_like(b)
    assert p.lib.tlr_factor_solve_c128(p.ctx, len(b), b.ctypes.data, x.ctypes.data) == 0
    return x


def _errors(K, b, x):
    """Normwise and rowwise backward error over the right-hand sides."""
    aK = np.abs(K).astype(float)
    norm, row = [], []
    for bv, xv in zip(b, x):
        r = np.abs(bv - K @ xv.astype(K.dtype)).astype(float)
        norm.append(np.linalg.norm(r) / (np.linalg.norm(aK) * np.linalg.norm(xv)))
        row.append(np.linalg.norm(r / (aK @ np.abs(xv) + np.abs(bv))))
    return np.linalg.norm(norm), np.linalg.norm(row)


def _range(kind, decades, n, rng):
    span = lambda *s: 10.0 ** rng.uniform(-decades / 2, decades / 2, s)  # noqa: E731
    if kind == "entries":
        return span(n, n)
    if kind == "blocks":
        return np.kron(span(n // 10, n // 10), np.ones((10, 10)))
    return span(n, 1) if kind == "rows" else span(1, n)


@pytest.mark.parametrize("kind,decades", [("entries", 0), ("entries", 4), ("entries", 9),
                                          ("entries", 16), ("blocks", 12), ("rows", 6),
                                          ("columns", 12)])
def test_pencil(gpu_lib, kind, decades):
    n = 200
    rng = np.random.default_rng(decades)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A *= _range(kind, decades, n, rng)
    b = rng.standard_normal((4, n)) + 1j * rng.standard_normal((4, n))
    with api.PencilProblem(A, np.eye(n), Physics(omega=0j, nev=1)) as p:
        sliced, fma = (_errors(A.astype(np.clongdouble), b, _solve(p, c, b)) for c in (0, 1))
    for s, f in zip(sliced, fma):
        assert 0 < s <= 3 * f


def test_grid(gpu_lib):
    ny, nz = 41, 23
    ph = Physics(alpha=2.7, reynolds=900.0, omega=0j, nev=1)
    with api.Problem(make_case(ny, nz, physics=ph)) as p:
        api.run_pipeline(p)

        def out(what, dtype):
            a = np.empty(p.lib.tlr_out_bytes(p.ctx, what) // np.dtype(dtype).itemsize, dtype)
            assert p.lib.tlr_copy_out(p.ctx, what, a.ctypes.data, a.nbytes) == 0
            return a

        nn = ny * nz
        col, blocks = out(3, np.int32).reshape(nn, -1), out(6, complex).reshape(nn, -1, 5, 5)
        K = np.zeros((5 * nn, 5 * nn), complex)
        for i in range(nn):
            for c, blk in zip(col[i], blocks[i]):
                K[5 * i:5 * i + 5, 5 * c:5 * c + 5] += blk
        rng = np.random.default_rng(1)
        b = rng.standard_normal((4, 5 * nn)) + 1j * rng.standard_normal((4, 5 * nn))
        K = K.astype(np.clongdouble)
        sliced, fma = (_errors(K, b, _solve(p, c, b)) for c in (0, 1))
    for s, f in zip(sliced, fma):
        assert 0 < s <= 3 * f

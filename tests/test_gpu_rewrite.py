"""The rewrite of a complex128 factor by the inverses of its diagonal blocks
(L' = L inv(L_bb) and U' = inv(U_bb) U in exact integer slices, D_b = inv(U_bb)
inv(L_bb) and blocks of fewer than 32 columns in FP64) against the FP64 products on the CUDA cores, on one front.

Sizes: one block and several, last blocks of 1, 33 and 44 rows (one to four
passes, a last pass of one column), no border and one of many tiles.  Both
multiply the same inverses, so they differ by the errors of the products alone:
the FP64 chain's, 2 (2 x 128 + 2) 2^-53 |A| |B|, and the slices', in each of up to
four passes 4 x 64 x 2^-55 of the largest terms (row maximum x column maximum
after the pivot scaling), with one FP64 addition per pass.  Against extended
precision the slices must not be worse in the norm (with a tenth to spare)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(lib, A, p, sliced):
    m = A.shape[0]
    front = np.ascontiguousarray(A.T).view(np.float64).reshape(-1)
    sizes = [min(128, p - b) for b in range(0, p, 128)]
    out = np.zeros_like(front)
    d = np.zeros(2 * sum(n * n for n in sizes))
    assert lib.tlr_rewrite_c128(front.ctypes.data, m, p, sliced, out.ctypes.data,
                                d.ctypes.data) == 0
    D, at = [], 0
    for n in sizes:
        D.append(d[at:at + 2 * n * n].view(np.complex128).reshape(n, n).T)
        at += 2 * n * n
    return out.view(np.complex128).reshape(m, m).T, D


def _factored(m, p, scaling, rng):
    A = rng.standard_normal((m, m)) + 1j * rng.standard_normal((m, m))
    if scaling != "one":
        A *= 10.0 ** rng.uniform(-6, 6, m)[:, None]
    if scaling == "lines":
        A *= 10.0 ** rng.uniform(-6, 6, m)[None, :]
    for k in range(p):
        q = k + int(np.argmax(np.abs(A[k:p, k])))
        A[[k, q]] = A[[q, k]]
        A[k + 1:, k] /= A[k, k]
        A[k + 1:, k + 1:] -= np.outer(A[k + 1:, k], A[k, k + 1:])
    return A


def _inverses(K):
    """Inverses of the unit lower and of the upper triangle in extended precision."""
    n = K.shape[0]
    K = K.astype(np.clongdouble)
    lo, up = np.eye(n, dtype=K.dtype), np.eye(n, dtype=K.dtype)
    for q in range(n):
        lo[q + 1:] -= np.outer(K[q + 1:, q], lo[q])
    for q in range(n - 1, -1, -1):
        up[q] /= K[q, q]
        up[:q] -= np.outer(K[:q, q], up[q])
    return lo, up


@pytest.mark.parametrize("scaling", ["one", "rows", "lines"])
@pytest.mark.parametrize("m,p", [(33, 33), (130, 129), (160, 40), (300, 300), (417, 161),
                                 (700, 128)])
def test_sliced_rewrite(gpu_lib, m, p, scaling):
    A = _factored(m, p, scaling, np.random.default_rng(m + p))
    got, gd = _run(gpu_lib, A, p, 1)
    ref, rd = _run(gpu_lib, A, p, 0)
    untouched = np.ones((m, m), bool)
    for t, b in enumerate(range(0, p, 128)):
        e = min(p, b + 128)
        untouched[e:, b:e] = untouched[b:e, e:] = False
        lo, up = _inverses(A[b:e, b:e])
        assert np.array_equal(gd[t], rd[t])
        products = []
        if e < m:
            products = [(A[e:, b:e], lo, got[e:, b:e], ref[e:, b:e]),
                        (up, A[b:e, e:], got[b:e, e:], ref[b:e, e:])]
        for X, Y, g, r in products:
            exact = X.astype(np.clongdouble) @ Y.astype(np.clongdouble)
            aX, aY = np.abs(X).astype(float), np.abs(Y).astype(float)
            s = np.max(aY, axis=1)
            if X is not up:  # L': scaled by the columns of L
                s = 1 / np.max(aX, axis=0)
            top = (np.max(aX * s, axis=1)[:, None] *
                   np.max(aY / np.where(s > 0, s, 1)[:, None], axis=0)[None, :])
            size = aX @ aY
            bound = (2 * 258 + 2 * 4) * 2.0 ** -53 * size + 4 * 4 * 64 * 2.0 ** -55 * top
            assert np.all(np.abs(g - r) <= bound)
            err, old = np.abs(g - exact).astype(float), np.abs(r - exact).astype(float)
            size = np.where(size > 0, size, 1)
            if e - b < 32:  # these blocks stay in FP64
                assert np.array_equal(g, r)
            assert np.sqrt(np.mean((err / size) ** 2)) <= 1.1 * np.sqrt(np.mean((old / size) ** 2))
    assert np.array_equal(got[untouched], A[untouched])


def test_nonfinite_entries(gpu_lib):
    """An infinite entry of L makes its row of L' not finite, and leaves the rest finite."""
    A = _factored(200, 100, "one", np.random.default_rng(5))
    A[150, 3] = np.inf
    got, _ = _run(gpu_lib, A, 100, 1)
    bad = ~np.isfinite(got)
    assert bad[150, :100].all()
    bad[150, :100] = False
    assert not bad.any()

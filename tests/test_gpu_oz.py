"""FP64 Schur update by exact integer slices on the tensor cores against
extended-precision NumPy and the CUDA-core FP64 kernel, on one front.

Sizes: remainders of the 128-row and 32-column tiles, a partial last panel,
one and many tiles.  Data: entries of one scale; pivot rows scaled over twelve
decades (as boundary rows against interior ones); rows and columns of their own
scale each.  A slice number carries 55 bits of its row's or column's largest
entry after the pivot scaling, the kept classes end 2^-64 below the largest
product, and F22 is rounded once, so the update's error, relative to |L21|
|U12| summed over the panel, stays within 64 x 2^-55 of the largest terms plus
half an ulp of the result.  The CUDA-core kernel rounds after every FMA; the
sliced one must not be worse in the norm (with a tenth to spare)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(lib, A, p, k0, sliced):
    m = A.shape[0]
    front = np.ascontiguousarray(A.T).view(np.float64).reshape(-1)
    out = np.zeros_like(front)
    st = lib.tlr_schur_update_c128(front.ctypes.data, m, p, k0, 32, sliced, out.ctypes.data)
    assert st == 0
    return out.view(np.complex128).reshape(m, m).T


@pytest.mark.parametrize("scaling", ["one", "pivots", "lines"])
@pytest.mark.parametrize("m,p,k0", [(33, 32, 0), (160, 64, 32), (203, 75, 64), (417, 100, 32),
                                    (700, 40, 0)])
def test_sliced_update(gpu_lib, m, p, k0, scaling):
    rng = np.random.default_rng(m + k0)
    A = rng.standard_normal((m, m)) + 1j * rng.standard_normal((m, m))
    b = min(p, k0 + 32)
    if scaling == "pivots":  # row k of U12 by d_k, column k of L21 by 1 / d_k
        d = 10.0 ** rng.uniform(-6, 6, b - k0)
        A[k0:b, b:] *= d[:, None]
        A[b:, k0:b] /= d[None, :]
    elif scaling == "lines":
        r, c = 10.0 ** rng.uniform(-8, 8, m - b), 10.0 ** rng.uniform(-8, 8, m - b)
        A[b:, k0:b] *= r[:, None]
        A[k0:b, b:] *= c[None, :]
        A[b:, b:] *= r[:, None] * c[None, :]
    L, U, C = A[b:, k0:b], A[k0:b, b:], A[b:, b:]
    ld = np.clongdouble
    exact = C.astype(ld) - L.astype(ld) @ U.astype(ld)
    size = np.abs(L) @ np.abs(U) + np.abs(C)
    got = _run(gpu_lib, A, p, k0, 1)
    ref = _run(gpu_lib, A, p, k0, 0)
    outside = got.copy()
    outside[b:, b:] = A[b:, b:]
    assert np.array_equal(outside, A)
    err = np.abs(got[b:, b:] - exact).astype(float) / size
    old = np.abs(ref[b:, b:] - exact).astype(float) / size
    assert np.sqrt(np.mean(err ** 2)) <= 1.1 * np.sqrt(np.mean(old ** 2))
    # largest terms: row maximum x column maximum after the pivot scaling
    e = np.max(np.abs(U), axis=1)
    top = np.max(np.abs(L) * e, axis=1)[:, None] * np.max(np.abs(U) / e[:, None], axis=0)[None, :]
    bound = 4 * 64 * 2.0 ** -55 * top + 2.0 ** -53 * np.abs(exact).astype(float)
    assert np.all(np.abs(got[b:, b:] - exact).astype(float) <= bound)


def test_nonfinite_entries_spread(gpu_lib):
    """An infinite entry of L21 or U12 makes its row or column of F22 not
    finite, and leaves the others finite."""
    rng = np.random.default_rng(3)
    A = rng.standard_normal((100, 100)) + 1j * rng.standard_normal((100, 100))
    A[50, 3] = np.inf
    A[5, 70] = np.nan
    got = _run(gpu_lib, A, 32, 0, 1)[32:, 32:]
    bad = np.zeros((68, 68), bool)
    bad[50 - 32, :] = True
    bad[:, 70 - 32] = True
    assert np.array_equal(~np.isfinite(got), bad)

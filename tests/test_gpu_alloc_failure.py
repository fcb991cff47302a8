"""A solve that runs out of memory leaves nothing half built: every allocation of
a mixed and of an FP64 solve fails once, on a fresh context, and the next solve on
the same context gives the eigenvalues of an undisturbed one.  Buffers that only
make a solve faster are not needed for it: without them it takes the path that
does without."""
import numpy as np
import pytest

from tailor_gb300 import api
from tailor_gb300.case import Physics, make_case

pytestmark = pytest.mark.gpu

NOMEM = (11, 12)  # TLR_ERR_CUDA with the allocation's message, TLR_ERR_NOMEM


# optional: allocations of the pipelined applications (15) and their solves (4), of
# the inverse form (8: these fronts have no second diagonal block, so the inversion
# needs no work space beyond the Schur updates'), of the slices of the FP64 form (4)
@pytest.mark.parametrize("precision,block,optional", [(1, 0, 27), (1, 2, 8), (0, 0, 4)])
def test_solve_after_a_failed_allocation(gpu_lib, precision, block, optional):
    ph = Physics(alpha=1.4, reynolds=700.0, nev=2, tol=1e-9)
    kw = dict(nev=2, ncv=12, precision=precision, block=block, fallback=False)

    def fresh():
        p = api.Problem(make_case(17, 12, physics=ph))
        api.run_pipeline(p)
        return p

    with fresh() as p:
        gpu_lib.tlr_alloc_fail_at(0)
        ref = api.EigenSolver(p).solve(**kw)
        count = gpu_lib.tlr_alloc_fail_at(0)
    assert count > 40
    failed = 0
    for k in range(1, count + 1):
        with fresh() as p:
            gpu_lib.tlr_alloc_fail_at(k)
            try:
                first = api.EigenSolver(p).solve(**kw)
                assert np.allclose(first.lam, ref.lam, rtol=1e-7, atol=0)
            except api.TailorError as e:
                assert e.status in NOMEM, e.message
                failed += 1
            finally:
                assert gpu_lib.tlr_alloc_fail_at(0) >= k
            again = api.EigenSolver(p).solve(**kw)
        assert np.allclose(again.lam, ref.lam, rtol=1e-7, atol=0)
    assert count - failed == optional


@pytest.mark.parametrize("precision,other", [(1, dict(cuda_core_schur=1)),
                                             (1, dict(persistent_solve=True)),
                                             (0, dict(cuda_core_schur=1))])
def test_no_buffers_of_another_form(gpu_lib, precision, other):
    """A factor makes the inverse form's or the slices' buffers only if it takes that
    form, on its first factorisation that does."""
    ph = Physics(alpha=1.4, reynolds=700.0, nev=2, tol=1e-9)
    kw = dict(nev=2, ncv=12, precision=precision, fallback=False)
    with api.Problem(make_case(17, 12, physics=ph)) as p:
        api.run_pipeline(p)
        lam, made = [], []
        for opts in (other, {}, other, {}):
            gpu_lib.tlr_alloc_fail_at(0)
            lam.append(api.EigenSolver(p).solve(**kw, **opts).lam)
            made.append(gpu_lib.tlr_alloc_fail_at(0))
    own = {1: 19 if "persistent_solve" in other else 0, 0: 0}[precision]
    assert made[1] - own == {1: 8, 0: 4}[precision]
    assert made[2:] == [0, 0]
    for a in lam[1:]:
        assert np.allclose(a, lam[0], rtol=1e-7, atol=0)

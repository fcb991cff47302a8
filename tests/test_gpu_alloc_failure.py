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


# optional: allocations of the pipelined applications (15) and their solves (4)
@pytest.mark.parametrize("precision,block,optional", [(1, 0, 19), (1, 2, 0), (0, 0, 0)])
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

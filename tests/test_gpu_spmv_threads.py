"""Products with host vectors by several threads on one problem: each gets its own
result (the calls share the context's stream and its device vectors)."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from tailor_gb300 import api
from tailor_gb300.case import make_case

pytestmark = pytest.mark.gpu


def test_concurrent_products(gpu_lib):
    with api.Problem(make_case(60, 32)) as p:
        api.run_pipeline(p)
        rng = np.random.default_rng(0)
        n = 5 * p.case.nodes
        xs = [rng.standard_normal(n) + 1j * rng.standard_normal(n) for _ in range(16)]
        ref = [p.spmv(api.TLR_MAT_A, x) for x in xs]
        with ThreadPoolExecutor(8) as pool:
            for _ in range(20):
                got = list(pool.map(lambda x: p.spmv(api.TLR_MAT_A, x), xs))
                for g, r in zip(got, ref):
                    assert np.array_equal(g, r)

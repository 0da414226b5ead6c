"""The expectation-value pass where its last warp or last CTA is partly
empty: pair counts around 32 and 128, n = 2 to 5, against the oracle with
the yardstick of its other tests."""
import numpy as np
import pytest

import oracle as orc
from ecg_b200 import Context
from test_gpu_expc import case_basis, close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [0, 1, "li_minus_like", "n5"])
@pytest.mark.parametrize("K", [1, 7, 8, 15, 16])
def test_partly_filled_warps_and_ctas(case, K):
    sysm, params = case_basis(case, K)
    rng = np.random.default_rng(K)
    c = rng.normal(size=K) + 1j * rng.normal(size=K)
    with Context(sysm, K, method="G") as ctx:
        ctx.set_params(params)
        ctx.compute_mat_elem(1, K, 0.0)
        gpu = ctx.expectation_values(K, -0.9, c, raw=True)
    o = orc.Oracle(sysm, K)
    o.set_params(params)
    o.compute_mat_elem(1, K, 0.0, method="G")
    close(gpu, o.expectation_values(K, c, -0.9), o.expectation_values(K, c, -0.9, extended=True), f"{case} K={K}")

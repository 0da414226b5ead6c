"""Whole factorisations of several sizes in one context: the cached graphs of
the persistent kernel share one array of tile counters, which stays where it
is when a larger size comes."""
import numpy as np
import pytest

from ecg_b200 import Context
from gpu_util import problem

pytestmark = pytest.mark.gpu


def solve(ctx, K, lam):
    ctx.set_vectors(K, last_eigvec=np.ones(K, dtype=np.complex128))
    E, err, it = ctx.energy_ia(1, K, lam, 1e-10)
    H, _, _, _, iD = ctx.matrices(K)
    return E, err, it, H, iD, ctx.vectors(K)[1]


@pytest.mark.parametrize("small,large", [(60, 65), (200, 700)])
def test_small_after_large_gives_the_small_result(small, large):
    """Small, large, small, large with allocations in between (the adjoint
    pass's and a candidate batch's buffers): bit for bit what a fresh context
    gives for each."""
    sysm, params, lam, _ = problem(1, large)
    fresh = {}
    for K in (small, large):
        with Context(sysm, large + 1) as ctx:
            ctx.set_params(params)
            fresh[K] = solve(ctx, K, lam)
    with Context(sysm, large + 1) as ctx:
        ctx.set_params(params)
        for K in (small, large, small, large, small):
            got = solve(ctx, K, lam)
            assert got[:3] == fresh[K][:3], K
            assert all(np.array_equal(a, b) for a, b in zip(got[3:], fresh[K][3:])), K
            if K == large:
                ctx.energy_ib_adjoint(0, K, lam, 1e-10)
                ctx.set_vectors(K + 1, last_eigvec=np.ones(K + 1, dtype=np.complex128))
                ctx.eval_candidates(K, params[:20] * 1.01, lam, 1e-10)

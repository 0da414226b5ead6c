"""Bounded waits that run out where no other wait can do so first: the call
reports ECG_ECUDA, and after the limit is restored the context gives what it
gave before, bit for bit."""
import numpy as np
import pytest

from ecg_b200 import Context, EcgError
from gpu_util import problem
from test_gpu_candidates import base_problem

pytestmark = pytest.mark.gpu
ECG_ECUDA = -2


@pytest.mark.parametrize("K0", [8, 40, 64])
def test_candidates_gemm_copies(K0):
    """A base of one panel: its solves wait for no other panel, so the first
    wait a limit of 0 ends is that of the GEMM for its bulk copies, with
    copies in flight."""
    tol = 1e-10
    sysm, params, cands, _, lam, start = base_problem(1, K0, 30, 7, tol)

    def batch(ctx):
        ctx.set_vectors(K0 + 1, last_eigvec=start)
        return ctx.eval_candidates(K0, cands, lam, tol)

    with Context(sysm, K0 + 1) as ctx:
        ctx.set_params(params)
        ctx.set_vectors(K0, last_eigvec=np.ones(K0, dtype=np.complex128))
        ctx.energy_ia(1, K0, lam, tol)
        E0, err0, it0, _ = batch(ctx)
        ctx.set_wait_limit(0)
        with pytest.raises(EcgError) as ei:
            batch(ctx)
        assert ei.value.status == ECG_ECUDA
        ctx.set_wait_limit(-1)
        E1, err1, it1, _ = batch(ctx)
    assert np.array_equal(E0, E1, equal_nan=True) and np.array_equal(err0, err1) and np.array_equal(it0, it1)


@pytest.mark.parametrize("K", [130, 400])
def test_iteration_solves(K):
    """A factorisation by one launch per panel step has no waits, so those of
    GHEPIIS's triangular solves run out first."""
    sysm, params, lam, _ = problem(1, K)

    def solve(ctx):
        ctx.set_vectors(K, last_eigvec=np.ones(K, dtype=np.complex128))
        return ctx.energy_ia(1, K, lam, 1e-10) + (ctx.vectors(K)[1],)

    with Context(sysm, K) as ctx:
        ctx.set_factor_mode(1)
        ctx.set_params(params)
        before = solve(ctx)
        ctx.set_wait_limit(0)
        with pytest.raises(EcgError) as ei:
            solve(ctx)
        assert ei.value.status == ECG_ECUDA
        ctx.set_wait_limit(-1)
        after = solve(ctx)
    assert after[:3] == before[:3] and np.array_equal(after[3], before[3])

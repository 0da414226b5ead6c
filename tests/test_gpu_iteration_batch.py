"""Inverse iterations enqueued several at a time: whatever number the last
call took, a call gives bit for bit what it gives in a fresh context, for
fewer and more iterations than that number, both stopping rules, every
normalisation and a MaxIter that cuts the iteration; a zero pivot leaves the
vectors alone."""
import numpy as np
import pytest

from ecg_b200 import Context
from gpu_util import problem

pytestmark = pytest.mark.gpu

K = 150


def solve(ctx, lam, tol, max_iter, norm):
    ctx.set_vectors(K, last_eigvec=np.ones(K, dtype=np.complex128))
    E, err, it = ctx.energy_ia(1, K, lam, tol, max_iter, specif_norm=norm)
    return E, err, it, ctx.vectors(K)[1]


@pytest.mark.parametrize("norm", [-1, 0, 1])
def test_results_do_not_depend_on_the_batch(norm):
    sysm, params, lam0, _ = problem(1, K)
    # near the eigenvalue (a few iterations), below the spectrum (many), cut
    # by MaxIter, the negative tolerance's rule, no iteration at all
    calls = [(lam0, 1e-10, 20), (lam0 - 0.5, 1e-8, 200), (lam0 - 0.5, 1e-8, 3), (lam0, 1e-2, 20), (lam0, -1e-6, 30),
             (lam0 - 0.5, 1e-13, 1), (lam0, 1e-10, 0), (lam0 - 0.1, 1e-10, 50)]
    fresh = []
    for lam, tol, m in calls:
        with Context(sysm, K) as ctx:
            ctx.set_params(params)
            fresh.append(solve(ctx, lam, tol, m, norm))
    with Context(sysm, K) as ctx:
        ctx.set_params(params)
        for order in (range(len(calls)), reversed(range(len(calls)))):
            for i in order:
                got = solve(ctx, *calls[i], norm)
                assert got[:3] == fresh[i][:3] and np.array_equal(got[3], fresh[i][3]), calls[i]
    assert len({f[2] for f in fresh}) >= 5  # different numbers of iterations were met


def test_zero_pivot_keeps_the_vector():
    """H - lambda S with a zero row: ErrorCode 1, no iteration, the starting
    vector and its normalisation untouched, and the context works on."""
    sysm, params, lam0, _ = problem(1, K)
    x0 = np.arange(1, K + 1) + 0.5j
    with Context(sysm, K) as ctx:
        ctx.set_params(params)
        E0, err0, it0, v0 = solve(ctx, lam0, 1e-10, 20, 0)
        H, S, dS, dH, _ = ctx.matrices(K)
        Z = np.zeros((K, K), dtype=np.complex128)
        ctx.set_matrices(H=Z, S=S, diagS=dS, diagH=np.zeros(K))
        ctx.set_vectors(K, last_eigvec=x0)
        E, err, it = ctx.energy_ia(1, K, 0.0, 1e-10, 1, mat_elem_needed=False, specif_norm=0)
        assert err == 1 and it == 0
        assert np.array_equal(ctx.vectors(K)[1], x0)
        again = solve(ctx, lam0, 1e-10, 20, 0)
    assert again[:3] == (E0, err0, it0) and np.array_equal(again[3], v0)

"""One new function beside a factorised basis (the trial loops): its row of H
and S from the row kernel, and the bordered factorisation as one forward
solve, at the edges of the 64-row panels, against the whole computation."""
import numpy as np
import pytest

from ecg_b200 import Context, synth
from gpu_util import problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg,n0,rows", [(0, 1, 1), (0, 33, 8), (1, 40, 9), (1, 63, 1), (1, 64, 1), (4, 200, 3)])
def test_rows_equal_the_whole_assembly(cfg, n0, rows):
    """ComputeMatElem(n0+1, n0+rows) after ComputeMatElem(1, n0) leaves bit
    for bit the matrices of ComputeMatElem(1, n0+rows) (8 rows at most take
    the row kernel, 9 the tiles), and so do the tile entry points."""
    K = n0 + rows
    sysm, params = synth.config_basis(cfg, K=K)
    with Context(sysm, K) as a, Context(sysm, K) as b, Context(sysm, K) as c:
        for ctx in (a, b, c):
            ctx.set_params(params)
        a.compute_mat_elem(1, K, -1.1)
        b.compute_mat_elem(1, n0, -1.1)
        b.compute_mat_elem(n0 + 1, K, -1.1)
        c.compute_mat_elem(1, n0, -1.1)
        c.compute_mat_elem_tiles(n0 + 1, K, -1.1, 0, c.pair_tiles(n0 + 1, K))
        ref = a.matrices(K)
        for ctx in (b, c):
            got = ctx.matrices(K)
            for x, y in zip(got[:3], ref[:3]):
                assert np.array_equal(np.tril(x) if x.ndim == 2 else x, np.tril(y) if y.ndim == 2 else y)
            assert np.array_equal(got[1], ref[1])


@pytest.mark.parametrize("K", [3, 4, 64, 65, 66, 129, 200])
@pytest.mark.parametrize("pivot_mode", [0, 1])
def test_bordered_row_matches_the_whole_factorisation(K, pivot_mode):
    """EnergyIA(K, K) beside the factor of K - 1 rows against EnergyIA(1, K):
    below the spectrum, where M = H - lambda S is well conditioned, the new
    column of L^H and its pivot agree to rounding (1e-11 of the largest
    entry), and a second trial in the same row starts from the same factor.
    Energies are stationary: 1e-12."""
    sysm, params, lam0, _ = problem(1, K)
    other = synth.random_basis(sysm.n, 1, 77)
    lam = lam0 - 0.5
    ones = np.ones(K, dtype=np.complex128)

    def solve(ctx, nmin):
        ctx.set_vectors(K, last_eigvec=ones)
        E, err, _ = ctx.energy_ia(nmin, K, lam, 1e-10, 200)
        H, _, _, _, iD = ctx.matrices(K)
        return E, err, np.triu(H, 1), iD

    with Context(sysm, K) as a, Context(sysm, K) as b:
        for ctx in (a, b):
            ctx.set_pivot_mode(pivot_mode)
            ctx.set_params(params)
        E0, err0, U0, iD0 = solve(a, 1)
        b.set_vectors(K, last_eigvec=ones)
        b.energy_ia(1, K - 1, lam, 1e-10, 200)
        b.set_params(other, first=K)
        solve(b, K)
        b.set_params(params[K - 1:], first=K)
        E1, err1, U1, iD1 = solve(b, K)
    assert err0 == err1 and abs(E0 - E1) <= 1e-12 * abs(E0)
    assert np.max(np.abs(U1 - U0)) <= 1e-11 * max(1.0, np.max(np.abs(U0)))
    assert np.max(np.abs(iD1 - iD0)) <= 1e-11 * np.max(np.abs(iD0))


@pytest.mark.parametrize("cfg,K", [(0, 33), (1, 65), (4, 96), ("4n4", 40)])
def test_gradient_of_one_function(cfg, K):
    """EnergyIB(K-1, K) sums the newest function's row on its own: its
    gradient is the last part of EnergyIB(0, K)'s (1e-11 of the largest
    entry: the same pairs in another order)."""
    sysm, params, lam, _ = problem(cfg, K)
    ones = np.ones(K, dtype=np.complex128)
    with Context(sysm, K) as ctx:
        ctx.set_params(params)
        ctx.set_vectors(K, last_eigvec=ones)
        E, err, _ = ctx.energy_ia(1, K, lam, 1e-13, 50, specif_norm=0)
        _, g, _, _ = ctx.energy_ib_adjoint(0, K, lam, 1e-13, 50)
        _, g1, _, _ = ctx.energy_ib_adjoint(K - 1, K, lam, 1e-13, 50)
    assert np.max(np.abs(g1 - g[-sysm.npt:])) <= 1e-11 * np.max(np.abs(g))

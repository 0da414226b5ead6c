"""The persistent LDL^H factorisation at the edges of its tiles and of its
task list: sizes around one 8-row block, one 64-row panel, the first update
of two, three and four panels at once, and the first update that is one task
of the list for four panels (a tile row 8 or more beyond the group's first
panel: nine panels, a last panel of one row, of 63 and of 64)."""
import numpy as np
import pytest

from ecg_b200 import Context
from gpu_util import problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pivot_mode", [0, 1])
@pytest.mark.parametrize("K", [2, 7, 8, 9, 63, 65, 72, 127, 128, 129, 191, 193, 257, 321, 449, 513, 575, 576, 577, 641,
                               833, 900])
def test_factor_reproduces_the_matrix(K, pivot_mode):
    """max |U^H D U - M| <= 1e-12 max |M| below the spectrum, where M = H -
    lambda S is definite: the bound of an elimination without growth is
    about 4 K eps = 8e-13 at the largest K here."""
    sysm, params, lam0, _ = problem(1, K)
    with Context(sysm, K) as ctx:
        ctx.set_pivot_mode(pivot_mode)
        ctx.set_params(params)
        ctx.set_vectors(K, last_eigvec=np.ones(K, dtype=np.complex128))
        ctx.energy_ia(1, K, lam0 - 0.5, 1e-12)
        H, _, _, _, iD = ctx.matrices(K)
    M = np.tril(H) + np.tril(H, -1).conj().T
    U = np.triu(H, 1) + np.eye(K)
    R = U.conj().T @ ((1.0 / iD)[:, None] * U)
    assert np.max(np.abs(R - M)) <= 1e-12 * np.max(np.abs(M))

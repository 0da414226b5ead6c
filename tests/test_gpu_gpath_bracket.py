"""EnergyGA's bracket before the inverse iteration: a narrow one around the
last call's eigenvalue, the few halvings of a first call, and the further
ones a dense part of the spectrum takes, against LAPACK's generalised
eigenvalues of the same matrices."""
import numpy as np
import pytest
import scipy.linalg

from ecg_b200 import Context, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg,K", [(1, 30), (1, 64), (1, 150), (4, 100)])
@pytest.mark.parametrize("which", [1, 2, 5, 9])
def test_eigenvalue_from_every_kind_of_bracket(cfg, K, which):
    """Both sides lose about cond(S) eps of the eigenvalue: a factor of 32 on
    it, from S's own condition number."""
    sysm, params = synth.config_basis(cfg, K=K)
    with Context(sysm, K, method="G") as ctx:
        ctx.set_params(params)
        first, err, nf = ctx.energy_ga(1, K, which=which, want_vector=True)
        H, S, _, dH, _ = ctx.matrices(K)
        again, err2, nf2 = ctx.energy_ga(1, K, which=which)
        ctx.set_params(params * (1.0 + 1e-7))
        moved, err3, nf3 = ctx.energy_ga(1, K, which=which)
        Hm, Sm, _, dHm, _ = ctx.matrices(K)
    assert err == err2 == err3 == 0
    for E, h, s, d in ((first, H, S, dH), (again, H, S, dH), (moved, Hm, Sm, dHm)):
        h = np.tril(h) + np.tril(h, -1).conj().T
        s = np.tril(s) + np.tril(s, -1).conj().T
        np.fill_diagonal(h, d)  # the diagonals are kept apart
        np.fill_diagonal(s, 1.0)
        ref = scipy.linalg.eigh(h, s, eigvals_only=True)[which - 1]
        tol = 32 * np.finfo(float).eps * np.linalg.cond(s) * max(1.0, abs(ref))
        assert abs(E - ref) <= tol, (E, ref, tol)
    assert nf2 <= nf and nf3 <= nf

"""EnergyGA where an eigenvalue lies just outside the narrow bracket around
the last call's energy: the inverse iteration at the bracket's centre then
gains almost nothing a step, and a residual that stands still is not the
iteration's floor."""
import numpy as np
import pytest

from ecg_b200 import Context, synth

pytestmark = pytest.mark.gpu


def load(ctx, n, lam, theta):
    """H = diag(lam, 5, 6, ...), its first two axes turned by theta, S = 1."""
    H = np.diag(np.arange(n) + 3.0).astype(np.complex128)
    c, s = np.cos(theta), np.sin(theta)
    R = np.array([[c, -s], [s, c]])
    H[:2, :2] = R @ np.diag(lam) @ R.T
    ctx.set_matrices(H=H, S=np.zeros((n, n)), diagS=np.ones(n), diagH=np.diag(H).real.copy())


@pytest.mark.parametrize("n", [2, 40, 70])
@pytest.mark.parametrize("l1,l2", [(-1 + 0.98e-6, -1 + 1.01e-6), (-1 + 0.9e-6, -1 + 1.06e-6), (-1 + 0.5e-6, -1 + 1.1e-6)])
def test_neighbour_outside_the_warm_bracket(n, l1, l2):
    """Start vector 3e-6 off the eigenvector.  The matrix is rounded to a few
    eps, which turns the eigenvector by that over the gap; the iteration's
    own residual adds its tolerance: 8 eps / (l2 - l1) + 1e-10."""
    theta = 3e-6
    sysm, _ = synth.config_basis(1, K=2)
    with Context(sysm, n, method="G") as ctx:
        load(ctx, n, (-1.0, -0.5), 0.0)
        E, err, _ = ctx.energy_ga(1, n, want_vector=True, mat_elem_needed=False)
        assert err == 0 and abs(E + 1.0) <= 1e-14
        load(ctx, n, (l1, l2), theta)
        E, err, nf = ctx.energy_ga(1, n, want_vector=True, mat_elem_needed=False)
        v, _ = ctx.vectors(n)
    assert err == 0 and abs(E - l1) <= 1e-14
    off = abs(-np.sin(theta) * v[0] + np.cos(theta) * v[1]) / np.linalg.norm(v)
    bound = 8 * np.finfo(float).eps / (l2 - l1) + 1e-10
    print(f"n {n}: off by {off:.2e} of {bound:.2e}, {nf} factorisations")
    assert off <= bound

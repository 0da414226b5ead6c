"""EnergyGA on an unchanged basis, where the bisection meets the eigenvalue itself."""
import pytest

from ecg_b200 import Context, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,seed", [(60, s) for s in range(6)])
def test_solving_the_same_basis_again(K, seed):
    """EnergyGA called again on an unchanged basis bisects first at the
    eigenvalue itself, where rounding decides the inertia count: the energy
    of every call is the first one's (within 1e-12), not the centre of the
    last bracket (about 1e-9 away)."""
    sysm, _ = synth.config_basis(1, K=K)
    with Context(sysm, K, method="G") as ctx:
        ctx.set_params(synth.random_basis(sysm.n, K, 500 + seed))
        first, err, _ = ctx.energy_ga(1, K)
        assert err == 0
        for _ in range(4):
            E, err, _ = ctx.energy_ga(1, K)
            assert err == 0 and abs(E - first) <= 1e-12 * abs(first), (E, first)

"""Factorisations by launches with 6000 new rows or more take their panels in
pairs: whole ones in factor mode 1, with an even and an odd number of panels,
and a border of that many rows beside an existing factor."""
import numpy as np
import pytest

from ecg_b200 import Context, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,first", [(6100, 0), (6020, 0), (6150, 100)])
def test_energy_and_eigenvector_against_the_persistent_kernel(K, first):
    """Both forms lose a few K eps of the largest |H| entry over the gap; the
    energies within the 1e-10 of the comparison with the oracle, the
    eigenvector within 1e-8, as at smaller sizes."""
    sysm, params = synth.config_basis(2, K=K)
    with Context(sysm, K) as ctx:
        ctx.set_params(params)
        ones = np.ones(K, dtype=np.complex128)
        ctx.set_vectors(K, last_eigvec=ones)
        E0, _, _ = ctx.energy_ia(1, K, synth.SYSTEMS["h2_like"]["e_floor"], -1e-12, max_iter=300, specif_norm=0)
        lam = E0 * 1.000001
        out = []
        for mode in (0, 1):
            ctx.set_factor_mode(mode)
            ctx.set_vectors(K, last_eigvec=ones)
            if mode and first:
                ctx.energy_ia(1, first, lam, 1e-10)
                ctx.set_vectors(K, last_eigvec=ones)
                E, err, it = ctx.energy_ia(first + 1, K, lam, 1e-11, specif_norm=0)
            else:
                E, err, it = ctx.energy_ia(1, K, lam, 1e-11, specif_norm=0)
            out.append((E, err, it, ctx.vectors(K)[1]))
    (Ep, errp, itp, xp), (El, errl, itl, xl) = out
    dx = np.max(np.abs(xp - xl)) / np.max(np.abs(xl))
    print(f"K {K}: E {Ep:.15f} {El:.15f} codes {errp} {errl} iterations {itp} {itl} eigenvector {dx:.1e}")
    assert errp == errl == 0 and abs(Ep - El) <= 1e-10 and dx <= 1e-8

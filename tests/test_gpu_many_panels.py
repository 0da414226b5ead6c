"""Bases grown function by function have a panel for each; beyond the
co-resident CTAs a step of the inverse iteration is a launch per panel."""
import numpy as np
import pytest

from ecg_b200 import Context
from gpu_util import problem

pytestmark = pytest.mark.gpu


def test_no_surplus_steps_after_many_iterations():
    """340 panels.  A call from a poor start vector, then one from the
    solution: the second launches only what its own few iterations take, and
    both give the energy of the basis in whole panels."""
    K, first, tol = 360, 20, 1e-10
    sysm, params, lam0, _ = problem(1, K)
    lam = lam0 - 0.1
    start = np.cos(np.arange(K)).astype(np.complex128)
    with Context(sysm, K) as ctx:
        ctx.set_params(params)
        ctx.set_vectors(K, last_eigvec=start)
        E0, err0, _ = ctx.energy_ia(1, K, lam, tol, 100)
    with Context(sysm, K) as ctx:
        ctx.set_params(params)
        ctx.set_vectors(K, last_eigvec=start)
        ctx.energy_ia(1, first, lam, tol, 100)
        for k in range(first + 1, K):
            ctx.energy_ia(k, k, lam, tol, 1)
        got, before = [], ctx.launch_count()
        for v in (start, None):
            if v is not None:
                ctx.set_vectors(K, last_eigvec=v)
            E, err, it = ctx.energy_ia(K, K, lam, tol, 100)
            now = ctx.launch_count()
            got.append((E, err, it, now - before))
            before = now
    (Ea, erra, ita, la), (Eb, errb, itb, lb) = got
    print(f"E {E0:.15f} {Ea:.15f} {Eb:.15f}, iterations {ita} {itb}, launches {la} {lb}")
    assert err0 == erra == errb == 0 and ita >= itb + 4
    assert abs(Ea - E0) <= 1e-10 and abs(Eb - E0) <= 1e-10
    nb = K - first + 1  # the first rows are one panel
    assert la - lb >= (ita - itb) * 2 * nb

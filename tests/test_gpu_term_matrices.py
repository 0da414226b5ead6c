"""Pair terms under every kind of term matrix P, n = 2..5: all products of
particle transpositions (identity, exchanges that do and do not move the
reference particle, cycles of both), whose congruence P Z P' is made of
additions and swaps, and integer matrices that are none, which take the
general product.  Derivatives with respect to both functions against the
oracle."""
import itertools

import numpy as np
import pytest

import oracle as orc
from ecg_b200 import Context, System, synth
from gpu_util import term_conditions, tolerance

pytestmark = pytest.mark.gpu


def particle_permutation(perm):
    """Matrix on the n relative coordinates r_i = R_i - R_0 of R_x -> R_perm[x]."""
    n = len(perm) - 1
    P = np.zeros((n, n), dtype=np.int32)
    for i in range(n):
        if perm[i + 1]:
            P[i, perm[i + 1] - 1] += 1
        if perm[0]:
            P[i, perm[0] - 1] -= 1
    return P


def term_matrices(n):
    perms = list(itertools.permutations(range(n + 1)))
    rng = np.random.default_rng(n)
    if len(perms) > 60:
        perms = perms[:1] + [perms[i] for i in sorted(rng.choice(np.arange(1, len(perms)), 56, replace=False))]
    mats = [particle_permutation(p) for p in perms]
    shear = np.eye(n, dtype=np.int32)
    shear[0, 1] = 1
    both = -np.eye(n, dtype=np.int32)
    both[0, 1] = 2
    return np.array(mats + [shear, both, 2 * np.eye(n, dtype=np.int32)], dtype=np.int32)


@pytest.mark.parametrize("n", [2, 3, 4, 5])
def test_every_term_matrix(n):
    sysm = System([3.0 + i for i in range(n + 1)], [1.0] + [-1.0] * n, "1")
    mats = term_matrices(n)
    sysm.yhy_mats, sysm.yhy_coeffs, sysm.T = mats, np.ones(len(mats), dtype=np.int32), len(mats)
    rng = np.random.default_rng(100 + n)
    basis = synth.random_basis(n, 32, seed=5)
    terms = np.repeat(np.arange(len(mats)), 3).astype(np.int32)
    pk, pl = basis[rng.integers(0, 32, terms.size)], basis[rng.integers(0, 32, terms.size)]
    o = orc.Oracle(sysm, 4)
    with Context(sysm, 4) as ctx:
        H, S, Dk, Dl = ctx.matrix_elements(pk, pl, terms, 3)
    tol = tolerance(term_conditions(sysm, pk, pl, terms), c=256.0)  # as tests/test_gpu_pair_elements.py
    worst = 0.0
    for i, t in enumerate(terms):
        h, s, dk, dl = o.matrix_elements(pk[i], pl[i], mats[t], 3)
        e = max(abs(H[i] - h) / max(abs(h), abs(s)), abs(S[i] - s) / abs(s),
                np.max(np.abs(Dk[i] - dk)) / np.max(np.abs(dk)), np.max(np.abs(Dl[i] - dl)) / np.max(np.abs(dl)))
        worst = max(worst, e / tol[i])
    print(f"n={n}: {len(mats)} matrices, worst diff/tolerance {worst:.3f}")
    assert worst <= 1.0

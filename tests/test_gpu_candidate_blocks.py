"""Batched candidates at the edges of the triangular solves' blocks: batches
that run in 16-column blocks (more than 256) against the same candidates in
batches small enough for 8-column blocks, bases of 1 to 3 panels with a last
panel of 1, 31, 33, 63 and 64 rows, and a base grown row by row, whose
panels are irregular."""
import numpy as np
import pytest

from ecg_b200 import Context, synth
from gpu_util import problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbase,count,grown", [(1, 257, 0), (31, 257, 0), (33, 320, 0), (64, 258, 0), (65, 257, 0),
                                               (127, 300, 0), (129, 257, 0), (70, 257, 5), (130, 300, 3), (100, 20100, 0), (700, 300, 0)])
def test_batches_of_both_widths_agree(nbase, count, grown):
    """Below the spectrum, where the iteration is well conditioned, the two
    widths multiply and add the same numbers in the same order except in the
    GEMM, whose inner sum is cut into pieces by the number of tiles (from
    pieces of one chunk to several tiles a piece): energies agree to 1e-11
    (a stationary value of vectors converged to 1e-9), ErrorCodes exactly."""
    sysm, params, lam0, _ = problem(1, nbase)
    cands = synth.candidates(params, count, 5)
    lam = lam0 - 0.5
    with Context(sysm, nbase + 1) as ctx:
        ctx.set_params(params)
        ctx.set_vectors(nbase + 1, last_eigvec=np.ones(nbase + 1, dtype=np.complex128))
        ctx.energy_ia(1, nbase - grown, lam, 1e-9, 400)
        for k in range(nbase - grown + 1, nbase + 1):
            ctx.energy_ia(k, k, lam, 1e-9, 400)
        start = np.ones(nbase + 1, dtype=np.complex128)
        ctx.set_vectors(nbase + 1, last_eigvec=start)
        E, err, _, _ = ctx.eval_candidates(nbase, cands, lam, 1e-9, 400)
        parts = [ctx.eval_candidates(nbase, cands[i:i + 50], lam, 1e-9, 400) for i in range(0, count, 50)]
    assert np.array_equal(err, np.concatenate([p[1] for p in parts]))
    Ep = np.concatenate([p[0] for p in parts])
    ok = err == 0
    assert ok.any() and np.max(np.abs(E[ok] - Ep[ok])) <= 1e-11

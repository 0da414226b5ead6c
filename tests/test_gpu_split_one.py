"""The adjoint partials of one function by ranges of tiles: every value that a
pass over more functions writes is written, so that a buffer the caller did
not clear can be summed or exchanged as a whole."""
import numpy as np
import pytest
import torch

from ecg_b200 import Context
from gpu_util import problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg,K", [(1, 2), (1, 32), (1, 33), (1, 97), (2, 75), (4, 40)])
def test_every_partial_of_one_function_is_written(cfg, K):
    sysm, params, lam, _ = problem(cfg, K)
    with Context(sysm, K) as ctx:
        ctx.set_params(params)
        ctx.set_vectors(K, last_eigvec=np.ones(K, dtype=np.complex128))
        ctx.energy_ia(1, K, lam, 1e-10)
        E, g0, err, _ = ctx.energy_ib_adjoint(K - 1, K, lam, 1e-10)
        assert err == 0
        nt, pd = ctx.pair_tiles(K, K), ctx.adjoint_part_doubles()
        buf = torch.full((nt * pd,), float("nan"), dtype=torch.float64, device="cuda:0")
        ctx.adjoint_tiles(K - 1, K, E, 0, nt, buf.data_ptr())
        g = ctx.adjoint_finish(K - 1, K, buf.data_ptr())
    assert np.array_equal(g, g0)
    p = buf.cpu().numpy().reshape(nt, 2, 32, -1)  # tile, rows and columns, slot, value
    slot = (K - 1) % 32
    rows = np.delete(p[:, 0], slot, axis=1)
    assert np.all(np.isfinite(p[:, 0, slot])) and np.all(rows == 0.0)
    assert np.all(p[-1, 1, slot:] == 0.0)  # the last tile holds the function's own column

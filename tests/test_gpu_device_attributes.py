"""The kernels' shared-memory limits belong to the device's context, not to
the process: with a new one (here after the device was reset, as on a second
device) every kernel still launches."""
import os
import subprocess
import sys

import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import ctypes, sys
import numpy as np
from ecg_b200 import Context, synth

K = 90
sysm = synth.make_system("li_minus_like")
params = synth.random_basis(sysm.n, K, 3, row_scale=synth.reduced_mass_scale(sysm.masses))

def evaluate():
    out = []
    for mode in (0, 1):
        with Context(sysm, K + 1, max_nfo=K) as ctx:
            ctx.set_factor_mode(mode)
            ctx.set_params(params)
            for fn in (ctx.energy_ib_adjoint, ctx.energy_ib):
                ctx.set_vectors(K, last_eigvec=np.ones(K, dtype=np.complex128))
                E, g, err, it = fn(0, K, -9.0, 1e-8, 100)
                out += [np.array([E, err, it], dtype=float), g]
            ctx.set_vectors(K + 1, last_eigvec=np.ones(K + 1, dtype=np.complex128))
            E, err, it, ra, g = ctx.eval_candidates_grad(K, params[:9] * 1.02, -9.0, 1e-8, 100)
            out += [E, err, g]
    return out

first = evaluate()
assert ctypes.CDLL("libcudart.so.12").cudaDeviceReset() == 0
again = evaluate()
assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(first, again))
print("same")
"""


def test_results_after_a_new_device_context():
    env = dict(os.environ, PYTHONPATH=PKG + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", SCRIPT], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr[-2000:]

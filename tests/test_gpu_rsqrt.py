"""The branch-free reciprocal square root of the pair terms (ecg_math.cuh)
and what is built on it, against extended precision.

Bounds, in units u = 2^-53 relative: the last rounding is 1 u, the rounding
of x y inside e = 1 - x y^2 reaches the result halved (0.5 u), the series'
remainder is below 2^-60: 2 u for rsqrt_series.  1/b squares it (4 u), with
the squared modulus's own rounding (1.5 u) and two products (2 u): 8 u of
the modulus.  1/sqrt(a) takes half of 1/a's error, another rsqrt_series and
three products: 12 u of the modulus."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(__file__), "..", "atom-mol-nonbo_b200", "csrc")
SOURCE = r"""
#include "ecg_math.cuh"
using namespace ecg;
__global__ void k(const double* x, int n, double* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const cd z = mk(x[2 * i], x[2 * i + 1]);
    cd inv;
    const cd is = crsqrt(z, inv), r = crcp_series(z);
    double* o = out + 7 * (size_t)i;
    o[0] = rsqrt_series(fabs(z.x));
    o[1] = is.x; o[2] = is.y; o[3] = inv.x; o[4] = inv.y; o[5] = r.x; o[6] = r.y;
}
extern "C" int run(const double* x, int n, double* out)
{
    k<<<(n + 127) / 128, 128>>>(x, n, out);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("rsqrt")
    (d / "p.cu").write_text(SOURCE)
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", CSRC, "-shared",
                    "-Xcompiler", "-fPIC", "-o", str(d / "p.so"), str(d / "p.cu")], check=True)
    lib = C.CDLL(str(d / "p.so"))

    def call(z):
        x = torch.from_numpy(np.ascontiguousarray(z).view(np.float64).copy()).cuda()
        out = torch.zeros(7 * z.size, dtype=torch.float64, device="cuda")
        assert lib.run(C.c_void_p(x.data_ptr()), z.size, C.c_void_p(out.data_ptr())) == 0
        return out.cpu().numpy().reshape(-1, 7)

    return call


@pytest.mark.parametrize("decades", [0.5, 8, 70])
def test_accuracy(run, decades):
    rng = np.random.default_rng(int(decades))
    n = 100_000
    m = 10.0 ** rng.uniform(-decades, decades, n)
    a = rng.uniform(-np.pi, np.pi, n)
    a[:1000] = rng.choice([0.0, 1e-9, np.pi / 2, -np.pi / 2, np.pi - 1e-9], 1000)
    z = m * np.exp(1j * a)
    o = run(z)
    u = 2.0 ** -53
    zl = z.astype(np.clongdouble)
    x = np.abs(z.real)
    ok = x > 0
    r = 1.0 / np.sqrt(x[ok].astype(np.longdouble))
    e0 = np.max(np.abs(o[ok, 0] - r) / r)
    inv = 1.0 / zl
    e1 = np.max(np.abs((o[:, 3] + 1j * o[:, 4]) - inv) / np.abs(inv))
    e2 = np.max(np.abs((o[:, 5] + 1j * o[:, 6]) - inv) / np.abs(inv))
    sq = np.sqrt(inv)  # principal branch
    e3 = np.max(np.abs((o[:, 1] + 1j * o[:, 2]) - sq) / np.abs(sq))
    print(f"decades {decades}: rsqrt {e0 / u:.2f} u, 1/z {e1 / u:.2f} and {e2 / u:.2f} u, 1/sqrt(z) {e3 / u:.2f} u")
    assert e0 <= 2 * u and e1 <= 8 * u and e2 <= 8 * u and e3 <= 12 * u


def test_squared_modulus_beyond_the_range(run):
    """1/b where |b|^2 over- or underflows: zero-like and huge, never NaN."""
    o = run(np.array([1e200 + 1e190j, 1e-200 + 1e-210j]))
    assert np.all(np.isfinite(o[:, 5:7])) and abs(o[0, 5]) < 1e-100 and abs(o[1, 5]) > 1e100

"""The short reciprocal, quotient and root of the face fluxes (ff_device.cuh)
against 80-bit arithmetic, to the bounds their comments state, over magnitudes
far beyond those the fluxes meet, and rcp_any at the ends of the range."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from finflo_b200 import gpu

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SRC = r"""
#include "ff_device.cuh"
__global__ void k(const double* a, const double* b, double* o, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  o[i] = rcp(b[i]);
  o[n + i] = rcp_any(b[i]);
  o[2 * n + i] = quot(a[i], b[i], rcp(b[i]));
  sqrt_rsq(fabs(b[i]), o[3 * n + i], o[4 * n + i]);
}
extern "C" int math_run(const void* a, const void* b, void* o, int n) {
  k<<<(n + 127) / 128, 128>>>((const double*)a, (const double*)b, (double*)o, n);
  return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("math")
    (d / "math.cu").write_text(SRC)
    csrc = os.path.join(os.path.dirname(gpu.__file__), "csrc")
    subprocess.check_call(["nvcc"] + gpu.NVCC_FLAGS + ["-I", csrc, "-o", str(d / "math.so"), str(d / "math.cu")])
    L = ctypes.CDLL(str(d / "math.so"))
    L.math_run.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int]

    def f(a, b):
        da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
        o = torch.empty(5, len(a), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert L.math_run(da.data_ptr(), db.data_ptr(), o.data_ptr(), len(a)) == 0
        return o.cpu().numpy()
    return f


def _ulps(got, ref):
    """Error of got in units of its own last place, ref in 80 bits."""
    return float((np.abs(got.astype(np.longdouble) - ref) / np.spacing(np.abs(got))).max())


def test_errors_against_80_bits(run):
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("long double is not 80 bits wide here")
    rng = np.random.default_rng(1)
    n = 1 << 21
    m = rng.uniform(1.0, 2.0, (2, n))
    m[:, :4096] = 1.0 + np.spacing(1.0) * np.arange(4096)            # mantissas next to the powers of two
    m[:, 4096:8192] = 2.0 - np.spacing(1.0) * np.arange(1, 4097)
    a, b = np.ldexp(m * rng.choice([-1.0, 1.0], (2, n)), rng.integers(-200, 200, (2, n)))
    r, ra, q, s, rs = run(a, b)
    A, B = a.astype(np.longdouble), b.astype(np.longdouble)
    assert _ulps(r, 1 / B) <= 0.507
    np.testing.assert_array_equal(ra, r)
    assert _ulps(q, A / B) <= 0.5005
    assert _ulps(s, np.sqrt(np.abs(B))) <= 0.5005
    assert _ulps(rs, 1 / np.sqrt(np.abs(B))) <= 1.005


def test_ends_of_the_range(run):
    b = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 4.0])
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(run(np.ones_like(b), b)[1], 1.0 / b)

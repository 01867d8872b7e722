"""The FP64 reciprocals, quotients and inverse roots that start from FP32
(mod_gemm.cuh) against IEEE division and square root."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "mod_gemm.cuh"
using namespace rimp2;
__global__ void k(const double *v, const double *d, double *out, int *odd, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  out[t] = recip_f64(d[t]);
  out[n + t] = div_f64(v[t], d[t]);
  bool o1 = false, o2 = false;
  out[2 * n + t] = recip_pos(fabs(d[t]), o1);
  out[3 * n + t] = rsqrt_pos(fabs(d[t]), o2);
  odd[t] = o1 || o2;
}
extern "C" int run(const double *v, const double *d, double *out, int *odd, int n) {
  double *dv, *dd, *dout;
  int *dodd;
  if (cudaMalloc(&dv, 8l * n) || cudaMalloc(&dd, 8l * n) || cudaMalloc(&dout, 32l * n) || cudaMalloc(&dodd, 4l * n)) return 1;
  cudaMemcpy(dv, v, 8l * n, cudaMemcpyHostToDevice);
  cudaMemcpy(dd, d, 8l * n, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(dv, dd, dout, dodd, n);
  cudaMemcpy(out, dout, 32l * n, cudaMemcpyDeviceToHost);
  const int rc = cudaMemcpy(odd, dodd, 4l * n, cudaMemcpyDeviceToHost);
  cudaFree(dv); cudaFree(dd); cudaFree(dout); cudaFree(dodd);
  return rc;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    from rimp2_gpu_gb300 import build
    d = tmp_path_factory.mktemp("div")
    src, so = str(d / "div.cu"), str(d / "div.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    cmd = [build.nvcc(), "-shared", src, "-o", so, "-I" + build.CSRC] + build._flags()
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(os.path.abspath(so))

    def call(v, d):
        n = len(d)
        out, odd = np.zeros((4, n)), np.zeros(n, dtype=np.int32)
        p = lambda x: x.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
        assert lib.run(p(v), p(d), p(out), p(odd), n) == 0
        return out, odd
    return call


def ulps(a, b):
    """Representable numbers between a and b of one sign."""
    return np.abs(a.view(np.int64) - b.view(np.int64))


def test_against_ieee(run):
    """The last step of each rounds once an error below 2^-64 (reciprocal, quotient)
    or 2^-53 (inverse root: d y rounded): within one number of the rounded value."""
    rng = np.random.default_rng(0)
    n = 1 << 20
    frac = 1.0 + rng.random(n)
    frac[: n // 8] = 1.0 + (np.arange(n // 8) - n // 16) % 4096 * 2.0 ** -52  # around powers of two
    frac[n // 8: n // 4] = 2.0 - (1 + np.arange(n // 8) % 4096) * 2.0 ** -52
    d = np.ldexp(frac, rng.integers(-110, 111, n)) * rng.choice([-1.0, 1.0], n)
    v = np.ldexp(1.0 + rng.random(n), rng.integers(-600, 601, n)) * rng.choice([-1.0, 1.0], n)
    v[::7] = d[::7] * np.ldexp(1.0, rng.integers(-9, 10, len(d[::7])))  # exact quotients
    out, odd = run(v, d)
    assert not odd.any()
    assert ulps(out[0], 1.0 / d).max() <= 1
    assert ulps(out[1], v / d).max() <= 1
    assert (out[1][::7] == v[::7] / d[::7]).all()
    assert ulps(out[2], 1.0 / np.abs(d)).max() <= 1
    root = (1.0 / np.sqrt(np.abs(d).astype(np.longdouble))).astype(np.float64)
    assert ulps(out[3], root).max() <= 1


def test_extremes(run):
    """Zeros, infinities, NaN, subnormals and large ratios are IEEE's own results; the
    inverse root and the positive reciprocal say that they are out of their range."""
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -2e-308, 1e-300, 1e300, 1.7e308, 3.0, -1e-37, 1e38, 1e-39])
    v, d = (np.ascontiguousarray(a.ravel()) for a in np.meshgrid(x, x))
    out, odd = run(v, d)
    with np.errstate(all="ignore"):
        for got, want in ((out[0], 1.0 / d), (out[1], v / d)):
            nan = np.isnan(want)
            assert (np.isnan(got) == nan).all()
            special = ~nan & (~np.isfinite(want) | (want == 0.0))
            assert (got[special] == want[special]).all()
            assert (np.signbit(got[special]) == np.signbit(want[special])).all()
            rest = ~nan & ~special
            assert ulps(got[rest], want[rest]).max() <= 1
    a = np.abs(d)
    out_of_range = ~((a >= 2.0 ** -1021) & (a < 2.0 ** 1018))
    assert (odd.astype(bool) == out_of_range).all()

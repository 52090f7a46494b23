"""The FP64 reciprocal of the lens kernels and of the critical curves' sums
(rcp_f64) against the correctly rounded quotient. The function has no entry
point; a kernel around it is compiled here."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from irs_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "shoot.cuh"
__global__ void rcp_kernel(const double* d, double* r, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) r[i] = irsb::rcp_f64(d[i]);
}
extern "C" int rcp_all(const double* host_d, double* host_r, int n) {
  double *d = nullptr, *r = nullptr;
  const size_t bytes = size_t(n) * sizeof(double);
  bool ok = cudaMalloc(&d, bytes) == cudaSuccess && cudaMalloc(&r, bytes) == cudaSuccess &&
            cudaMemcpy(d, host_d, bytes, cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok) rcp_kernel<<<592, 256>>>(d, r, n);
  ok = ok && cudaGetLastError() == cudaSuccess && cudaMemcpy(host_r, r, bytes, cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(d);
  cudaFree(r);
  return ok ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def rcp(gpu, tmp_path_factory):
    d = tmp_path_factory.mktemp("rcp")
    (d / "rcp.cu").write_text(SOURCE)
    out = str(d / "librcp.so")
    subprocess.run([build.nvcc()] + build.NVCC_FLAGS + ["-I", build.CSRC, str(d / "rcp.cu"), "-o", out], check=True,
                   capture_output=True)
    lib = ctypes.CDLL(out)

    def f(x):
        x = np.ascontiguousarray(x, np.float64)
        r = np.empty_like(x)
        assert lib.rcp_all(x.ctypes.data_as(ctypes.c_void_p), r.ctypes.data_as(ctypes.c_void_p), x.size) == 0
        return r
    return f


def test_reciprocal_within_its_bound(rcp):
    """The seed's relative error e is at most 2^-19; the step leaves e^3 <= 2^-57,
    1/16 ulp where the ulp is smallest against the value (2^-53), and rounds once:
    0.5 + 1/16 ulp, so at most one ulp from the rounded quotient. Mantissas random
    and at both ends, exponents over the range whose results are normal."""
    rng = np.random.default_rng(5)
    mant = np.concatenate([1 + rng.random(400000), 1 + 2.0 ** -52 * np.arange(200), 2 - 2.0 ** -52 * np.arange(1, 200)])
    exps = np.concatenate([rng.integers(-1022, 1021, mant.size - 6), [-1022, -1, 0, 1, 52, 1020]])
    d = np.ldexp(mant, exps) * rng.choice([-1.0, 1.0], mant.size)
    d = np.concatenate([d, mant])
    r = rcp(d)
    exact = 1.0 / d
    assert np.all(np.abs(r - exact) <= np.spacing(np.abs(exact)))
    if np.finfo(np.longdouble).nmant >= 63:  # the error itself, to 2^-10 ulp
        ld = np.longdouble
        err = np.abs(ld(1) - r.astype(ld) * d.astype(ld)) / np.abs(d.astype(ld)) / np.spacing(np.abs(r)).astype(ld)
        assert float(err.max()) <= 0.5 + 1 / 16 + 2.0 ** -10
        assert float(np.mean(r != exact)) < 0.1


def test_reciprocal_outside_its_range(rcp):
    """Zero, subnormal, infinite and NaN arguments give NaN; a result below the
    normal range is flushed to zero."""
    tiny = np.finfo(np.float64).tiny
    bad = np.array([0.0, -0.0, tiny / 2, -tiny / 4, 5e-324, np.inf, -np.inf, np.nan])
    assert np.all(np.isnan(rcp(bad)))
    big = np.ldexp(np.array([1.5, 1.999, -1.25]), 1022)
    assert np.all(rcp(np.concatenate([big, np.ldexp(np.array([1.0, 1.75]), 1023)])) == 0.0)
    assert rcp(np.array([tiny]))[0] == 1.0 / tiny

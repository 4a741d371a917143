"""The point physics' reciprocal and inverse square root (sint_physics.cuh)
against CUDA's division and rsqrt and against 64-bit mantissas on the host
(needs a B200 and nvcc).

Bounds: with a seed error e <= 2^-18 the series leave e^3 <= 2^-54, the last
operation rounds by 2^-53, and the inverse square root's e carries the rounding
of x y, 2^-53, of which half enters: below 2^-52 in FP64.  FP32: e^2 <= 2^-40,
the same roundings at 2^-24: below 2^-23.  CUDA's division rounds once, its
rsqrt is within one ulp.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "sint_physics.cuh"

template <typename R>
__global__ void both(int n, const R *x, R *out)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  out[i]         = sint::rcp_pos<R>(x[i]);
  out[n + i]     = sint::rsqrt_pos<R>(x[i]);
  out[2 * n + i] = R(1) / x[i];
  out[3 * n + i] = sizeof(R) == 8 ? R(rsqrt(double(x[i]))) : R(rsqrtf(float(x[i])));
}

extern "C" int run(int n, const void *x, void *out, int f64)
{
  const int blocks = (n + 255) / 256;
  if (f64)
    both<double><<<blocks, 256>>>(n, static_cast<const double *>(x), static_cast<double *>(out));
  else
    both<float><<<blocks, 256>>>(n, static_cast<const float *>(x), static_cast<float *>(out));
  const cudaError_t e = cudaGetLastError();
  return int(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("reciprocals")
    src, lib = d / "reciprocals.cu", d / "libreciprocals.so"
    src.write_text(SOURCE)
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-Xcompiler", "-fPIC", "-shared", "-I", os.path.join(ROOT, "hpsint_b200", "csrc"), "-o", str(lib),
                    str(src)], check=True)
    f = ctypes.CDLL(str(lib)).run
    f.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int]
    return f


# FP64: the callers' squared norms start at 1e-20; up to where the reciprocal
# is still a normal number.  FP32: the normal results of normal arguments.
@pytest.mark.parametrize("dtype,lo,hi,ulp", [(np.float64, -20.0, 45.0, 2.0**-52), (np.float64, -300.0, 300.0, 2.0**-52),
                                             (np.float32, -20.0, 37.0, 2.0**-23)])
def test_reciprocals(run, dtype, lo, hi, ulp):
    rng = np.random.default_rng(7)
    x = np.concatenate([10.0**rng.uniform(lo, hi, 1 << 20), 2.0**np.arange(-60, 61),
                        np.nextafter(1.0, [0.0, 2.0]), 4.0 - 2.0**-np.arange(1.0, 24.0)]).astype(dtype)
    xd = torch.as_tensor(x, device="cuda")
    out = torch.empty((4, len(x)), dtype=xd.dtype, device="cuda")
    torch.cuda.synchronize()
    assert run(len(x), xd.data_ptr(), out.data_ptr(), int(dtype is np.float64)) == 0
    got, exact = out.cpu().numpy().astype(np.longdouble), x.astype(np.longdouble)
    for ours, cuda, want, their_ulps in ((got[0], got[2], 1 / exact, 0.5), (got[1], got[3], 1 / np.sqrt(exact), 2.0)):
        assert np.max(np.abs(ours / want - 1)) <= ulp
        assert np.max(np.abs(ours / cuda - 1)) <= (1 + their_ulps) * ulp

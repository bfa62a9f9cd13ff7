"""The functions of fp64_light.cuh on the GPU: the quotient, the eighth root
and the FP32 <-> FP64 conversions, on ordinary values, at the edges of their
ranges and on every value that takes the fallback, against exact results.

Bars, with u = 2^-53 (half an FP64 ulp, relative) and U = 2^-24:
- the quotient's seed is within 5 U (2 ulp of the reciprocal, the operand's
  rounding), one Newton step leaves 9e-14, and the corrected quotient is
  rounded once: one of the two neighbours of a / b, so within one ulp of the
  rounded quotient;
- the root's seed is within 4.7 U, so the dropped term 0.05 h^3, h = 8 x 4.7 U,
  is 6e-19; y^8 carries 7 u of rounding, an eighth of which reaches the
  result, which is rounded once more: 1.9 u, and the fallback's three
  functions (half, half and one ulp) 2.8 u."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U53 = 2.0 ** -53
SRC = r"""
#include "fp64_light.cuh"
__global__ void k(int what, const double* a, const double* b, double* y, int* odd, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  bool o = false;
  if (what == 0) y[i] = lesgo::div_light(a[i], b[i]);
  else if (what == 1) y[i] = lesgo::inv_root8(a[i]);
  else if (what == 2) y[i] = lesgo::widen_fast((float)a[i], o);
  else y[i] = (double)lesgo::narrow_fast(a[i], o);
  odd[i] = o;
}
extern "C" int run(int what, const double* a, const double* b, double* y, int* odd, int n) {
  double* d = nullptr;
  int* f = nullptr;
  const size_t s = n * sizeof(double);
  if (n < 1 || cudaMalloc(&d, 3 * s) != cudaSuccess || cudaMalloc(&f, n * sizeof(int)) != cudaSuccess) return 1;
  cudaMemcpy(d, a, s, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, s, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(what, d, d + n, d + 2 * n, f, n);
  cudaMemcpy(y, d + 2 * n, s, cudaMemcpyDeviceToHost);
  cudaMemcpy(odd, f, n * sizeof(int), cudaMemcpyDeviceToHost);
  const int e = cudaGetLastError() != cudaSuccess;
  cudaFree(d);
  cudaFree(f);
  return e;
}
"""


@pytest.fixture(scope="module")
def light(tmp_path_factory):
    from lesgo_gb300.build import CSRC, NVCC_FLAGS, nvcc
    d = tmp_path_factory.mktemp("light")
    (d / "t.cu").write_text(SRC)
    subprocess.run([nvcc(), *NVCC_FLAGS, "-I" + CSRC, "-shared", str(d / "t.cu"), "-o", str(d / "t.so")], check=True)
    lib = C.CDLL(os.fspath(d / "t.so"))

    def run(what, a, b=None):
        a = np.ascontiguousarray(a, np.float64)
        b = np.ascontiguousarray(np.ones_like(a) if b is None else b, np.float64)
        y, odd = np.empty_like(a), np.zeros(a.size, np.int32)
        p = lambda x: C.c_void_p(x.ctypes.data)
        assert lib.run(what, p(a), p(b), p(y), p(odd), a.size) == 0
        return y, odd.astype(bool)
    return run


def spread(lo, hi, n, seed):
    """n positive values, even over the logarithm, and both ends' neighbours."""
    r = np.random.default_rng(seed)
    x = np.exp2(r.uniform(lo, hi, n))
    e = np.array([2.0 ** lo, 2.0 ** hi])
    return np.concatenate([x, e, np.nextafter(e, 0), np.nextafter(e, np.inf)])


ODD = np.array([0.0, -0.0, 5e-324, -1e-310, 2.0 ** -1022, 2.0 ** -101, -2.0 ** 101, 1e300, np.inf, -np.inf, np.nan])


def test_quotient(light):
    a, b = spread(-99, 99, 100000, 1), spread(-99, 99, 100000, 2)[::-1]
    s = np.random.default_rng(3).choice([-1.0, 1.0], (2, a.size))
    a, b = a * s[0], b * s[1]
    y, _ = light(0, a, b)
    ref = a / b
    assert np.max(np.abs(y - ref) / np.spacing(np.abs(ref))) <= 1.0


def test_quotient_outside_its_range(light):
    """The device's division, which rounds correctly; a zero over an ordinary
    value is zero."""
    a, b = (x.ravel() for x in np.meshgrid(np.concatenate([ODD, [1.0, -3.0]]), np.concatenate([ODD, [1.0, 7.0]])))
    y, _ = light(0, a, b)
    with np.errstate(all="ignore"):
        assert np.array_equal(y, a / b, equal_nan=True)


def test_eighth_root(light):
    x = spread(-99, 99, 100000, 4)
    y, _ = light(1, x)
    ref = 1 / np.sqrt(np.sqrt(np.sqrt(x.astype(np.longdouble))))
    assert np.max(np.abs(y / ref - 1)) <= 2 * U53


def test_eighth_root_outside_its_range(light):
    x = np.array([5e-324, 1e-310, 2.0 ** -1022, 2.0 ** -101, 2.0 ** 100, 2.0 ** 101, 1e300])
    y, _ = light(1, x)
    ref = 1 / np.sqrt(np.sqrt(np.sqrt(x.astype(np.longdouble))))
    assert np.max(np.abs(y / ref - 1)) <= 3 * U53
    y, _ = light(1, np.array([0.0, np.inf, -1.0, -np.inf, np.nan]))
    assert y[0] == np.inf and y[1] == 0.0 and np.all(np.isnan(y[2:]))


def test_widen(light):
    x = spread(-126, 127, 50000, 5).astype(np.float32)
    x = np.concatenate([x, -x, [np.float32(3.4028235e38), np.float32(2.0 ** -126)]])
    x = x[np.abs(x) >= np.float32(2.0 ** -126)]
    y, odd = light(2, x.astype(np.float64))
    assert not odd.any() and np.array_equal(y, x.astype(np.float64))
    _, odd = light(2, np.array([0.0, -0.0, 1e-40, -1e-45, np.inf, -np.inf, np.nan]))
    assert odd.all()


def test_narrow(light):
    """Round to nearest even, ties and carries into the exponent among them."""
    x = spread(-125, 126, 50000, 6)
    up = x.astype(np.float32).astype(np.float64).view(np.uint64) & ~np.uint64(0x1fffffff)
    ties = (up | np.uint64(0x10000000)).view(np.float64)
    carry = np.nextafter(2.0 ** np.arange(-125, 127.0), 0)
    x = np.concatenate([x, ties, np.nextafter(ties, 0), np.nextafter(ties, np.inf), carry, [2.0 ** -126]])
    x = np.concatenate([x, -x])
    y, odd = light(3, x)
    assert not odd.any() and np.array_equal(y, x.astype(np.float32).astype(np.float64))
    _, odd = light(3, np.array([0.0, -0.0, np.nextafter(2.0 ** -126, 0), 1e-40, 5e-324, 2.0 ** 127, 1e39, np.inf,
                                -np.inf, np.nan]))
    assert odd.all()

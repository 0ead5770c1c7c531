"""The device forms of div_by (csrc/clb_div.h) and sincos_link (csrc/clb_trig.h), which the host tests of
both headers do not run: quotients bit for bit, sines and cosines against 80-bit ones, on both sides of
the change to the library's functions."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from cosmolattice_b200 import build

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.abspath(build.__file__)), "csrc")
NVCC = os.environ.get("NVCC", "nvcc")

SRC = r"""
#include "clb_div.h"
#include "clb_trig.h"
template <class T> __global__ void k_div(const T *x, T *q, int n, clb::DivBy d)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) q[i] = clb::div_by(x[i], d);
}
template <class T> __global__ void k_sincos(const T *x, T *s, T *c, int n)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) clb::sincos_link(x[i], &s[i], &c[i]);
}
template <class T> static int run(const T *x, T *a, T *b, int n, const clb::DivBy *d)
{
  T *p = nullptr;
  if (cudaMalloc(&p, 3 * sizeof(T) * n) != cudaSuccess) return 1;
  cudaMemcpy(p, x, sizeof(T) * n, cudaMemcpyHostToDevice);
  if (d)
    k_div<T><<<(n + 255) / 256, 256>>>(p, p + n, n, *d);
  else
    k_sincos<T><<<(n + 255) / 256, 256>>>(p, p + n, p + 2 * n, n);
  cudaMemcpy(a, p + n, sizeof(T) * n, cudaMemcpyDeviceToHost);
  if (b) cudaMemcpy(b, p + 2 * n, sizeof(T) * n, cudaMemcpyDeviceToHost);
  cudaFree(p);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
extern "C" {
int div64(const double *x, double *q, int n, double y) { const clb::DivBy d = clb::make_div(y, (float)y); return run(x, q, (double *)nullptr, n, &d); }
int div32(const float *x, float *q, int n, double y) { const clb::DivBy d = clb::make_div(y, (float)y); return run(x, q, (float *)nullptr, n, &d); }
int sincos64(const double *x, double *s, double *c, int n) { return run(x, s, c, n, (const clb::DivBy *)nullptr); }
int sincos32(const float *x, float *s, float *c, int n) { return run(x, s, c, n, (const clb::DivBy *)nullptr); }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which(NVCC) is None:
        pytest.skip("needs nvcc")
    d = tmp_path_factory.mktemp("device_math")
    (d / "t.cu").write_text(SRC)
    subprocess.run([NVCC, *build.NVCC_FLAGS, f"-I{CSRC}", "-shared", str(d / "t.cu"), "-o", str(d / "t.so")], check=True)
    return C.CDLL(str(d / "t.so"))


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("y", [2 * np.pi / 64, 2 * np.pi / 99, (2 * np.pi / 125) ** 2, 2.0 ** -7, 0.3, 17.5])
def test_div_by_on_the_device_gives_the_quotient_bits(lib, y):
    rng = np.random.default_rng(int(1e6 * y))
    n = 200000
    x = rng.uniform(1, 2, n) * 2.0 ** rng.integers(-200, 200, n) * rng.choice([-1, 1], n)
    # numerators whose quotient lies next to a half-way point between two doubles
    q = rng.uniform(1, 2, n // 2)
    x[: n // 2] = np.nextafter((q + q * 2.0 ** -53) * y, rng.choice([0.0, 4.0 * y], n // 2))
    x[0] = 0.0
    out = np.empty(n)
    assert lib.div64(_ptr(x), _ptr(out), n, C.c_double(y)) == 0
    assert np.array_equal(out.view(np.uint64), (x / y).view(np.uint64))
    # a negative zero may lose its sign, and nothing else
    z = np.array([-0.0])
    assert lib.div64(_ptr(z), _ptr(out), 1, C.c_double(y)) == 0 and out[0] == 0
    # FP32 multiplies by the rounded divisor's reciprocal
    x32, out32 = (x[np.abs(np.log2(np.abs(x) + 1e-300)) < 60]).astype(np.float32), np.empty(n, np.float32)
    assert lib.div32(_ptr(x32), _ptr(out32), len(x32), C.c_double(y)) == 0
    want = x32 * (np.float32(1) / np.float32(y))
    assert np.array_equal(out32[: len(x32)].view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("dtype,fn", [(np.float64, "sincos64"), (np.float32, "sincos32")])
@pytest.mark.parametrize("lo,hi,ulps", [(1e-9, 1 / 32, 0.55), (1 / 32, 4.0, 2.0)])
def test_sincos_link_on_the_device(lib, dtype, fn, lo, hi, ulps):
    # up to 1/32 the polynomials (0.55 of the last place, as on the host), beyond it the CUDA library's
    # functions, whose documented bound is 2
    rng = np.random.default_rng(3)
    n = 300000
    x = (np.exp(rng.uniform(np.log(lo), np.log(hi), n)) * rng.choice([-1, 1], n)).astype(dtype)
    edge = dtype(1 / 32)
    x[:4] = [edge, -edge, np.nextafter(edge, dtype(0)), np.nextafter(edge, dtype(1))]
    x = x[(np.abs(x) <= edge) == (hi <= 1 / 32)]
    s, c = np.empty_like(x), np.empty_like(x)
    assert getattr(lib, fn)(_ptr(x), _ptr(s), _ptr(c), len(x)) == 0
    for got, want in ((s, np.sin(x.astype(np.longdouble))), (c, np.cos(x.astype(np.longdouble)))):
        w = want.astype(dtype)
        # the spacing of the numbers on the side of the true value
        ulp = np.where(np.abs(want) < np.abs(w), np.abs(w) - np.nextafter(np.abs(w), dtype(0)), np.nextafter(np.abs(w), dtype(10)) - np.abs(w))
        assert float((np.abs(got - want) / ulp).max()) <= ulps

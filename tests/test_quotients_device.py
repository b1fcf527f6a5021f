"""divc and div_n of csrc/cvlbm_math.cuh against the division, bit for bit but for the
sign of a zero quotient (and two units in the last place for numerators below 2^-968).

A kernel around the header's own functions, compiled here: operands over the whole
range of doubles, zeros of either sign, infinities and NaN, and divisors and numerators
on, just inside and just outside the limits of the short form.
"""

from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

SOURCE = r"""
#include <cuda_runtime.h>
#include <vector>
#include "cvlbm_math.cuh"
__global__ void k(int n, const cv::DivC* d, const double* a, const double* b, double* oc,
                  double* o1, double* o9) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  double v[9], w[9];
  for (int j = 0; j < 9; ++j) v[j] = a[9 * t + j];
  for (int j = 0; j < 9; ++j) oc[9 * t + j] = cv::divc(v[j], d[t]);
  const cv::Rcp r = cv::rcp_of(b[t]);
  cv::div_n(r, v, w, 9);
  for (int j = 0; j < 9; ++j) o9[9 * t + j] = w[j];
  for (int j = 0; j < 9; ++j) {  // groups of one: every numerator decides for itself
    cv::div_n(r, v + j, w, 1);
    o1[9 * t + j] = w[0];
  }
}
extern "C" int run(int n, const double* a, const double* b, double* out) {
  std::vector<cv::DivC> d(n);
  for (int t = 0; t < n; ++t) d[t] = cv::make_divc(b[t]);
  const size_t na = sizeof(double) * 9 * (size_t)n;
  cv::DivC* dd = nullptr;
  double *da = nullptr, *db = nullptr, *o = nullptr;
  if (cudaMalloc(&dd, sizeof(cv::DivC) * n) || cudaMalloc(&da, na) ||
      cudaMalloc(&db, sizeof(double) * n) || cudaMalloc(&o, 3 * na))
    return 1;
  cudaMemcpy(dd, d.data(), sizeof(cv::DivC) * n, cudaMemcpyHostToDevice);
  cudaMemcpy(da, a, na, cudaMemcpyHostToDevice);
  cudaMemcpy(db, b, sizeof(double) * n, cudaMemcpyHostToDevice);
  k<<<(n + 127) / 128, 128>>>(n, dd, da, db, o, o + 9 * (size_t)n, o + 18 * (size_t)n);
  const int rc = cudaMemcpy(out, o, 3 * na, cudaMemcpyDeviceToHost);
  cudaFree(dd); cudaFree(da); cudaFree(db); cudaFree(o);
  return rc;
}
"""


def _around(x):
    return [float(np.nextafter(x, 0.0)), x, float(np.nextafter(x, np.inf))]


def _operands():
    rng = np.random.default_rng(11)

    def randoms(n, lo, hi):
        v = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n))
        return v * rng.choice((-1.0, 1.0), n)

    special = [0.0, np.inf, np.nan, 5e-324, 2.0 ** -1074 * 3, 2.0 ** -1022, 1.7e308, 1.0, 1.5,
               2.0 - 2.0 ** -52]
    edge_a = _around(2.0 ** 900) + _around(2.0 ** -968) + _around(2.0 ** -900)
    edge_b = _around(2.0 ** 100) + _around(2.0 ** -100) + [3.0, 0.1, 6.0, 1.1, 2.0 * 1.1 / 512]
    b = [s * x for x in special + edge_b for s in (1.0, -1.0)]
    b = np.array(b * 40 + list(randoms(6000, -99, 99)) + list(randoms(2000, -1022, 1023)))
    pool = np.array([s * x for x in special + edge_a for s in (1.0, -1.0)])
    a = np.empty((b.size, 9))
    for t in range(b.size):
        if t % 3 == 0:  # edges and special values together
            a[t] = rng.choice(pool, 9)
        elif t % 3 == 1:  # a regular group with zeros among it
            a[t] = randoms(9, -860, 880)
            a[t, rng.integers(0, 9, 3)] = rng.choice((0.0, -0.0), 3)
        else:
            a[t] = randoms(9, -1074, 1023)
    return a, b


@pytest.mark.gpu
def test_quotients_on_the_device(tmp_path):
    from curved_lbm import _build

    src, lib = tmp_path / "quot.cu", tmp_path / "quot.so"
    src.write_text(SOURCE)
    subprocess.run([_build.nvcc_path(), *_build.ARCH_FLAGS, *_build.NVCC_FLAGS, "-I",
                    str(_build.CSRC), "-shared", "-o", str(lib), str(src)], check=True)
    a, b = _operands()
    out = np.empty((3,) + a.shape)
    p = C.POINTER(C.c_double)
    rc = C.CDLL(str(lib)).run(b.size, a.ctypes.data_as(p), b.ctypes.data_as(p),
                              out.ctypes.data_as(p))
    assert rc == 0
    with np.errstate(all="ignore"):
        want = a / b[:, None]
    tiny = (np.abs(a) < 2.0 ** -968) & (a != 0.0)
    for name, got in zip(("divc", "div_n of one", "div_n of nine"), out):
        nan = np.isnan(want)
        assert np.array_equal(np.isnan(got), nan), name
        far = np.abs(np.abs(got).view(np.int64) - np.abs(want).view(np.int64))
        wrong = (np.signbit(got) != np.signbit(want)) & (want != 0.0)
        wrong |= far > np.where(tiny, 2, 0)
        wrong &= ~nan
        i = np.argwhere(wrong)
        assert not len(i), (name, len(i), [(a[t, j].hex(), b[t].hex(), got[t, j].hex(),
                                            want[t, j].hex()) for t, j in i[:5]])

"""The reciprocal, quotient and root helpers of csrc/dg_dp.cuh against CUDA's operators: random mantissas over all
exponents (both parities, on both sides of the borders between the Newton iterations and the operators), and zeros,
subnormal numbers, infinities and NaN of both signs.

Bars, in units of the last place of the operator's correctly rounded result: the last correction of dp_rcp, dp_div and
dp_root's square root is exact to a small fraction of an ulp, so at most the neighbour; its short form rounds x y, 1 ulp,
after the ulp of y; its reciprocal is within one ulp and 1/sqrt(x), of two roundings, within two.  Outside the iterations' range,
zeros of quotients and special values are the operator's.
"""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "galaexi_gb300", "csrc")

HARNESS = r"""
#include "dg_dp.cuh"
#include <cstdio>
#include <cstring>
#include <vector>
using namespace gx;
// distance in representable numbers; numbers of different sign or only one NaN: far apart
__device__ unsigned long long ulps(double a, double b) {
  const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
  if (a != a || b != b) return (a != a && b != b) ? 0 : ~0ull;
  if ((x ^ y) < 0) return ~0ull;
  return x > y ? x - y : y - x;
}
__global__ void check(const double* X, const double* Y, int n, unsigned long long* worst) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const double x = X[t], y = Y[t];
  double r, q;
  const double root = dp_root<true>(x, r), brief = dp_root<false>(x, q);
  const unsigned long long d[5] = {ulps(dp_rcp(x), 1. / x), ulps(dp_div(x, y), x / y), max(ulps(r, 1. / sqrt(x)), ulps(q, r)),
                                   ulps(root, sqrt(x)), ulps(brief, sqrt(x))};
  for (int k = 0; k < 5; ++k) atomicMax(worst + k, d[k]);
}
int main() {
  std::vector<double> x, y;
  unsigned long long s = 88172645463325252ull;
  auto next = [&] { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; };
  auto make = [&](unsigned long long e) {
    const unsigned long long b = (next() & 0x800fffffffffffffull) | (e << 52);
    double d;
    memcpy(&d, &b, 8);
    return d;
  };
  const unsigned long long edge[] = {0, 1, 122, 123, 124, 522, 523, 524, 1022, 1023, 1024, 1522, 1523, 1921, 1922, 1923, 2046, 2047};
  for (unsigned long long e = 0; e < 2048; ++e)
    for (int k = 0; k < 64; ++k) {
      const double a = make(e), b = make(next() & 2047), c = make(edge[next() % 18]);
      x.push_back(a); y.push_back(b);
      x.push_back(a); y.push_back(c);
      x.push_back(c); y.push_back(a);
      x.push_back(a); y.push_back(make(e < 40 ? e : e - next() % 40));
    }
  const double special[] = {0., -0., 1. / 0., -1. / 0., 0. / 0., 5e-324, -5e-324, 1., -1., 4., 2e-308, 1.7e308};
  for (double a : special)
    for (double b : special) { x.push_back(a); y.push_back(b); }
  const int n = (int)x.size();
  double *dx, *dy;
  unsigned long long *dw, w[5] = {0, 0, 0, 0, 0};
  if (cudaMalloc(&dx, n * 8) || cudaMalloc(&dy, n * 8) || cudaMalloc(&dw, sizeof w)) return 1;
  if (cudaMemcpy(dx, x.data(), n * 8, cudaMemcpyHostToDevice) || cudaMemcpy(dy, y.data(), n * 8, cudaMemcpyHostToDevice) ||
      cudaMemset(dw, 0, sizeof w)) return 1;
  check<<<(n + 127) / 128, 128>>>(dx, dy, n, dw);
  if (cudaMemcpy(w, dw, sizeof w, cudaMemcpyDeviceToHost)) return 1;
  printf("%llu %llu %llu %llu %llu\n", w[0], w[1], w[2], w[3], w[4]);
  return 0;
}
"""


def test_helpers_against_cuda_operators(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, exe = tmp_path / "dp.cu", tmp_path / "dp"
    src.write_text(HARNESS)
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I", CSRC, str(src), "-o",
                    str(exe)], check=True, capture_output=True, timeout=600)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    rcp, div, rsqrt, root, short = (int(v) for v in out.split())
    assert rcp <= 1 and div <= 1 and rsqrt <= 3 and root <= 1 and short <= 3, (rcp, div, rsqrt, root, short)

// Per-element scales of the mesh for the fixed-point kernels of the FP64 form, at dg_set_mesh.
#include "dg_ctx.h"
#include "dg_volume_fx.cuh"

namespace {

using gx::fx64;

// largest (or smallest) of a block's non-negative doubles as their bits (NaN: above all)
__device__ void block_max(double x, unsigned long long* s) {
  unsigned long long v = (unsigned long long)__double_as_longlong(x);
  for (int k = 16; k; k >>= 1) {
    const unsigned long long o = __shfl_xor_sync(0xffffffffu, v, k);
    v = o > v ? o : v;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(s, v);
}
__device__ double larger(double a, double b) { return b <= a ? a : b; }  // keeps a NaN that comes second
__device__ double keep(double a, double b) { return a == a ? larger(a, b) : a; }

// MetL[e][kMetL] (dg_volume_fx.cuh); flags: bit 0 an element flatter than 2^8, bit 1 SurfElem n differs from the metric terms
// of an element's face nodes (Gauss-Lobatto nodes; +- by side and flip) by more than 4.5e-16 SurfElem somewhere.
// Memory bound: one block per element reads the geometry once.
__global__ void __launch_bounds__(128)
k_mesh_scales(const double* __restrict__ Met, const double* __restrict__ Fgeo, const int* __restrict__ E2S, int n, int gl,
              float* __restrict__ MetL, int* __restrict__ flags) {
  const int n2 = n * n, n3 = n2 * n, N = n - 1;
  constexpr int NW = 19;
  __shared__ unsigned long long big[NW];  // 0-2 |M_d|^2, 3-11 M_d,c^2, 12 SurfElem, 13 |sJ|, 14 1/|sJ|, 15 |n_c|, 16-18 |SurfElem n_c|
  if (threadIdx.x < NW) big[threadIdx.x] = 0ull;
  __syncthreads();
  const size_t e = blockIdx.x;
  const double* const m = Met + e * 10 * n3;
  double w[NW];
  for (int c = 0; c < NW; ++c) w[c] = 0.;
  for (int t = threadIdx.x; t < n3; t += blockDim.x) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      double s = 0.;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double x = m[(size_t)(3 * d + c) * n3 + t], a = x * x;
        s += a;
        w[3 + 3 * d + c] = keep(w[3 + 3 * d + c], a);
      }
      w[d] = keep(w[d], s);
    }
    const double sj = fabs(m[(size_t)9 * n3 + t]);
    w[13] = keep(w[13], sj);
    w[14] = keep(w[14], 1. / sj);
  }
  bool differs = false;
  for (int t = threadIdx.x; t < 6 * n2; t += blockDim.x) {
    const int ls = t / n2 + 1, ab = t - (ls - 1) * n2, a = ab % n, b = ab / n;
    const size_t side = E2S[(e * 6 + ls - 1) * 2];
    const int flip = E2S[(e * 6 + ls - 1) * 2 + 1];
    int p, q;
    gx::s2v2_inv(N, a, b, flip, ls, p, q);
    const double* const f = Fgeo + side * 10 * n2 + p + n * q;
    const double se = f[9 * n2];
    w[12] = keep(w[12], fabs(se));
    const int dir = ls == gx::L_XI_MINUS || ls == gx::L_XI_PLUS ? 0 : (ls == gx::L_ETA_MINUS || ls == gx::L_ETA_PLUS ? 1 : 2);
    const bool minus = gx::is_minus(ls);
    const double sg = (minus ? -1. : 1.) * (flip == 0 ? 1. : -1.);
    const int node = gx::face_node(n, ls, a, b, minus ? 0 : N);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      w[15] = keep(w[15], fabs(f[c * n2]));
      w[16 + c] = keep(w[16 + c], fabs(se * f[c * n2]));
      differs = differs || !(fabs(__dsub_rn(sg * se * f[c * n2], m[(size_t)(3 * dir + c) * n3 + node])) <= se * 4.5e-16);
    }
  }
#pragma unroll
  for (int c = 0; c < NW; ++c) block_max(w[c], &big[c]);
  if (__syncthreads_or(gl && differs) && threadIdx.x == 0) atomicOr(flags, 2);
  if (threadIdx.x != 0) return;
  auto at = [&](int c) { return __longlong_as_double((long long)big[c]); };
  bool fine = at(13) < 1e45 && at(14) < 1e45;
  for (int d = 0; d < 3; ++d) fine = fine && at(d) > 1e-90 && at(d) < 1e90;
  float* const l = MetL + e * gx::kMetL;
  for (int c = 0; c < 12; ++c)
    l[c] = !fine ? gx::kFxNoScale : (at(c) > 1e-90 ? (float)(0.5 * log2(at(c)) + 1e-5) : -150.f);
  const bool face = fine && at(12) > 1e-45 && at(12) < 1e45 && at(15) <= 1. + 1e-9;
  l[12] = face ? (float)(log2(at(12)) + 1e-5) : gx::kFxNoScale;
  l[13] = face ? (float)(log2(at(13)) + 1e-5) : gx::kFxNoScale;
  for (int c = 0; c < 3; ++c) {
    const float f = face && at(16 + c) > 1e-45 ? (float)(log2(at(16 + c)) + 1e-5) : -150.f;
    l[14 + c] = fmaxf(fmaxf(l[3 + c], f), fmaxf(l[6 + c], l[9 + c]));
  }
  if (fmaxf(l[0], fmaxf(l[1], l[2])) - fminf(l[0], fminf(l[1], l[2])) > 8.f) atomicOr(flags, 1);
}

}  // namespace

namespace gxc {

cudaError_t mesh_scales(const double* Met, const double* Fgeo, const int* E2S, int nElems, int n, bool gl, float* MetL,
                        int* flags) {
  if (nElems > 0) k_mesh_scales<<<nElems, 128>>>(Met, Fgeo, E2S, n, gl ? 1 : 0, MetL, flags);
  return cudaGetLastError();
}

}  // namespace gxc

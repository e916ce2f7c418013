// k_lift_fx: the BR1 lifting of the FP64 form on Gauss-Lobatto nodes (strong, non-conservative form) in block
// fixed-point arithmetic on the integer pipes (dg_fx.cuh).
//
// Lifting_VolInt_Nonconservative (src/dg/lifting_volint.t90:262-328), the BR1 surface part
// (lifting_fillflux.t90:39-103, 212-256, surfint.t90:591-725) and ProlongToFaceLifting of u, v, w, T (no flux
// reads the density gradient).  On Gauss-Lobatto nodes the surface term of a node on a face is
//   L_hat 0.5 SurfElem n (P_slave - P_master),   SurfElem n = +- M_dir of the element's own face node
// up to the round-off of the mesh's metric terms.  Where the two are equal to the last bits (EXACT, checked on
// the device for the mesh, k_mesh_scales: affine elements), the term is added to the reference derivative of the face's
// direction before the metric terms: y_dir += N(N+1)/4 (neighbour - own) on the plus face, (own - neighbour)
// on the minus face, L_hat = N(N+1)/2; otherwise it is added in FP64 by face-node threads with the face's own
// geometry.  The gradients are g_d = sJ sum_dir M_dir,d y_dir.
// k_lift spent 159 FP64 instructions per node on this (65 cycles each per warp and sub-partition); here they
// are integer multiply-adds at 2 cycles, and the FP64 pipe only converts the twelve results.
//
// Mapping: one element per block.  One thread per line and variable differentiates the line in registers,
// with the even and odd parts of the line (D is centro-antisymmetric), which halves the products; then the
// threads finish node by node.
#pragma once
#include "dg_fx.cuh"
#include "dg_kernels.cuh"
#include "dg_lines.cuh"
#include "dg_volume_fx.cuh"

namespace gx {

template <int NP> struct LiftFx {
  static constexpr int NT = (4 * NP * NP + 31) / 32 * 32;   // one thread per line and variable
  static constexpr int NPT = (NP * NP * NP + NT - 1) / NT;  // nodes per thread
  static constexpr size_t smem = sizeof(fx64) * 16 * NP * NP * NP;
  // blocks per SM: shared memory (16 n^3 words) and 80 registers per thread
  static constexpr int MINB = NP >= 9 ? 1 : (NP == 8 ? 3 : (NP == 7 ? 3 : (NP == 6 ? 5 : (NP == 5 ? 6 : 12))));
};
// D = D_even + D_odd on the first half of the nodes (rows i < n/2; odd n: the middle node is the last column
// of even and the last row of odd), digits times 2^sD: y(i) = A + B, y(N-i) = B - A with
// A = sum even(i,l) (x_l + x_(N-l)) (middle: x), B = sum odd(i,l) (x_l - x_(N-l)); jump: N(N+1)/4
template <int NP> struct LiftFxBasis {
  static constexpr int H = NP / 2, HE = (NP + 1) / 2;
  FxDig even[H][HE], odd[HE][H], jump;
  int sD;
};

// Elements that take the FP64 sums: those where a magnitude mag of u, v, w, T is outside 2^+-150 (zeros aside), and
// those with a temperature below 2^-4 to 2^-5 of the largest, which would be held in fewer bits than in FP64 (57 below
// the largest; a node a million times as hot cost the others' second derivatives seven digits).  The latter are
// found in the conversion and left for the nodes' pass: a minimum beside the maxima, or a branch at the conversion's
// barrier, took 2 to 6% of the kernels.
__device__ __forceinline__ bool lift_cold(double T, unsigned mag) { return (mag >> 20) > (fx_mag(T) >> 20) + 4u; }
__device__ __forceinline__ bool lift_fits(const unsigned* mag) {
  const unsigned lowest = (1022u - 150u) << 20, highest = (1022u + 150u) << 20;
  bool ok = true;
#pragma unroll
  for (int v = 0; v < 4; ++v) ok = ok && mag[v] < highest && (mag[v] == 0u || mag[v] > lowest);
  return ok;
}

// u, v, w, T in FP64 to X [4][n3], and the derivatives of the lines of all directions to Y [3][4][n3] (elements whose
// values do not fit one scale): the FP64 kernel's sums, by the block (N = 7, 16^3, all elements: the kernel 0.590 ms, as
// k_lift; node by node from global memory 0.773)
template <int NP, int NT>
__device__ __noinline__ void lift_lines_fp64(const double* Pe, const double* D, double* X, double* Y) {
  constexpr int n = NP, n2 = NP * NP, n3 = NP * NP * NP;
  __syncthreads();
#pragma unroll 1
  for (int t = threadIdx.x; t < 4 * n3; t += NT) {
    const int v = t / n3, node = t - v * n3;
    X[v * n3 + vsw<NP>(node)] = Pe[(v == 3 ? 5 : v + 1) * n3 + node];
  }
  __syncthreads();
#pragma unroll 1
  for (int t = threadIdx.x; t < 12 * n2; t += NT) {
    const int dv = t / n2, li = t - dv * n2, dir = dv >> 2, step = dir == 0 ? 1 : (dir == 1 ? n : n2);
    const int base = dir == 0 ? n * li : (dir == 1 ? (li % n) + n2 * (li / n) : li);
    const double* const Xv = X + (dv & 3) * n3;
    double x[n];
#pragma unroll
    for (int l = 0; l < n; ++l) x[l] = Xv[vsw<NP>(base + l * step)];
#pragma unroll 2
    for (int i = 0; i < n; ++i) {
      double y = 0.;
#pragma unroll
      for (int l = 0; l < n; ++l) y = y + D[i + n * l] * x[l];
      Y[dv * n3 + vsw<NP>(base + i * step)] = y;
    }
  }
  __syncthreads();
}
// a node's gradients (volume part) from its derivatives, g[d * 4 + v]; then those of all nodes in the derivatives' place
template <int NP>
__device__ __forceinline__ void lift_node_fp64(const double* Me, const double* Y, int node, double g[12]) {
  constexpr int n3 = NP * NP * NP;
  const double sj = Me[(size_t)9 * n3 + node];
#pragma unroll
  for (int c = 0; c < 12; ++c) g[c] = 0.;
#pragma unroll
  for (int dir = 0; dir < 3; ++dir)
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double m = sj * Me[(size_t)(3 * dir + d) * n3 + node];
#pragma unroll
      for (int v = 0; v < 4; ++v) g[d * 4 + v] = g[d * 4 + v] + m * Y[(dir * 4 + v) * n3 + vsw<NP>(node)];
    }
}
template <int NP, int NT>
__device__ __noinline__ void lift_nodes_fp64(const double* Me, double* Y) {
  constexpr int n3 = NP * NP * NP;
#pragma unroll 1
  for (int node = threadIdx.x; node < n3; node += NT) {
    double g[12];
    lift_node_fp64<NP>(Me, Y, node, g);
#pragma unroll
    for (int c = 0; c < 12; ++c) Y[c * n3 + vsw<NP>(node)] = g[c];
  }
}

// the gradients of a node, and their traces on the faces it lies on (ProlongToFaceLifting)
template <int NP>
__device__ __forceinline__ void put_gradients(const double g[12], int node, size_t e, const int* es, int nSides,
                                              double* __restrict__ Gvol, double* __restrict__ Gf) {
  constexpr int n = NP, n2 = NP * NP, n3 = NP * NP * NP, N = NP - 1;
  double* const G = Gvol + e * 15 * n3 + node;
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int v = 0; v < 4; ++v) G[(d * 5 + 1 + v) * n3] = g[d * 4 + v];
  const int i = node % n, j = (node / n) % n, k = node / n2;
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    int ls, a, b;
    if (!node_face<NP>(f, i, j, k, ls, a, b)) continue;
    const int side = es[2 * (ls - 1)], flip = es[2 * (ls - 1) + 1];
    int p, q;
    s2v2_inv(N, a, b, flip, ls, p, q);
    double* const gf = Gf + ((size_t)(flip == 0 ? 0 : 1) * nSides + side) * 15 * n2 + p + n * q;
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int v = 0; v < 4; ++v) gf[(d * 5 + 1 + v) * n2] = g[d * 4 + v];
  }
}

template <int NP, bool EXACT>
__global__ void __launch_bounds__(LiftFx<NP>::NT, LiftFx<NP>::MINB)
k_lift_fx(const double* __restrict__ Pvol, const double* __restrict__ Met, const float* __restrict__ MetL,
          const double* __restrict__ Pf, const double* __restrict__ Fgeo, const int* __restrict__ E2S, const __grid_constant__ LiftFxBasis<NP> lb,
          const double* __restrict__ D, double Lhat, int nSides, double* __restrict__ Gvol, double* __restrict__ Gf) {
  using C = LiftFx<NP>;
  constexpr int n = NP, n2 = NP * NP, n3 = NP * NP * NP, N = NP - 1, NT = C::NT, NPT = C::NPT;
  constexpr int H = LiftFxBasis<NP>::H, HE = LiftFxBasis<NP>::HE;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  fx64* const Y = reinterpret_cast<fx64*>(smem_raw);           // [3][4][n3]: derivatives
  FxDig* const X = reinterpret_cast<FxDig*>(Y + 12 * n3);      // [4][n3]: u, v, w, T
  __shared__ unsigned mag[4];
  __shared__ int es[12], cold;
  const int e = blockIdx.x, tid = threadIdx.x;
  if (tid < 4) mag[tid] = 0u;
  if (tid == 0) cold = 0;
  if (tid < 12) es[tid] = E2S[(size_t)e * 12 + tid];
  __syncthreads();
  const double* const Pe = Pvol + (size_t)e * 7 * n3;
  const double* const Me = Met + (size_t)e * 10 * n3;
  auto liftc = [](int v) { return v == 3 ? 5 : v + 1; };
  // the neighbour's trace of lifted variable v at face coordinates (a, b) of local side ls
  auto trace = [&](int ls, int a, int b) {
    const int side = es[2 * (ls - 1)], flip = es[2 * (ls - 1) + 1];
    int p, q;
    s2v2_inv(N, a, b, flip, ls, p, q);
    return Pf + ((size_t)(flip == 0 ? 1 : 0) * nSides + side) * 6 * n2 + p + n * q;
  };
  // ---- one scale per variable: the largest magnitude of the element and its neighbours' traces
  double x[NPT][4];
  {
    unsigned m[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int it = 0; it < NPT; ++it) {
      const int node = tid + it * NT;
      if (node < n3)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          x[it][v] = Pe[liftc(v) * n3 + node];
          m[v] = max(m[v], fx_mag(x[it][v]));
        }
    }
    if (EXACT) for (int t = tid; t < 6 * n2; t += NT) {
      const int ls = t / n2 + 1, pq = t - (ls - 1) * n2;
      const double* nb = Pf + ((size_t)(es[2 * (ls - 1) + 1] == 0 ? 1 : 0) * nSides + es[2 * (ls - 1)]) * 6 * n2 + pq;
#pragma unroll
      for (int v = 0; v < 4; ++v) m[v] = max(m[v], fx_mag(nb[liftc(v) * n2]));
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) fx_block_max(m[v], &mag[v]);
  }
  __syncthreads();
  const float* const ml = MetL + (size_t)e * kMetL;
  bool ok = ml[0] < 200.f && lift_fits(mag);
  if (ok) {
#pragma unroll
    for (int it = 0; it < NPT; ++it) {
      const int node = tid + it * NT;
      if (node < n3) {
#pragma unroll
        for (int v = 0; v < 4; ++v) X[v * n3 + vsw<NP>(node)] = fd_from(x[it][v], fx_r0(57 - fx_exp(mag[v])));
        if (lift_cold(x[it][3], mag[3])) cold = 1;
      }
    }
    __syncthreads();
    // ---- derivatives.  |x| < 2^57 and |D| < 2^58 in digits: a sum of at most 5 products of (x_l +- x_(N-l)) and D
    // stays below 2^63 in all partial sums, and y, in units of 2^(57 - e + sD - 60 + 3), below 2^61 (three more
    // bits than the digits' unit: |D| is up to 2^5, y of a smooth field far below the bound)
    if (tid < 4 * n2) {
      const int v = tid / n2, li = tid - v * n2;
      const FxDig* const Xv = X + v * n3;
      const int r0 = fx_r0(57 - fx_exp(mag[v]));
#pragma unroll 1
      for (int dir = 0; dir < 3; ++dir) {
        const int step = dir == 0 ? 1 : (dir == 1 ? n : n2);
        const int base = dir == 0 ? n * li : (dir == 1 ? (li % n) + n2 * (li / n) : li);
        const int lm = dir == 0 ? L_XI_MINUS : (dir == 1 ? L_ETA_MINUS : L_ZETA_MINUS);
        const int lp = dir == 0 ? L_XI_PLUS : (dir == 1 ? L_ETA_PLUS : L_ZETA_PLUS);
        double nm = 0., np = 0.;
        if constexpr (EXACT) {
          nm = trace(lm, li % n, li / n)[liftc(v) * n2];
          np = trace(lp, li % n, li / n)[liftc(v) * n2];
        }
        FxDig ev[HE], od[H], jm, jp;
#pragma unroll
        for (int l = 0; l < H; ++l) {
          const FxDig a = Xv[vsw<NP>(base + l * step)], b = Xv[vsw<NP>(base + (N - l) * step)];
          ev[l] = a + b;
          od[l] = a - b;
          if (EXACT && l == 0) {
            jm = a - fd_from(nm, r0);
            jp = fd_from(np, r0) - b;
          }
        }
        if constexpr (NP % 2) ev[H] = Xv[vsw<NP>(base + H * step)];
        fx64* const Yo = Y + (dir * 4 + v) * n3;
#pragma unroll
        for (int i = 0; i < H; ++i) {
          FxDot A, B;
#pragma unroll
          for (int l = 0; l < HE; ++l) {
            if (l == 4) A.carry();
            A.add(ev[l], lb.even[i][l]);
          }
#pragma unroll
          for (int l = 0; l < H; ++l) {
            if (l == 4) B.carry();
            B.add(od[l], lb.odd[i][l]);
          }
          const fx64 a = A.sum<3>(), b = B.sum<3>();
          fx64 y0 = a + b, yN = b - a;
          if (EXACT && i == 0) {
            FxDot j0, jN;
            j0.add(jm, lb.jump);
            jN.add(jp, lb.jump);
            y0 += j0.sum<3>();
            yN += jN.sum<3>();
          }
          Yo[vsw<NP>(base + i * step)] = y0;
          Yo[vsw<NP>(base + (N - i) * step)] = yN;
        }
        if constexpr (NP % 2) {
          FxDot B;
#pragma unroll
          for (int l = 0; l < H; ++l) B.add(od[l], lb.odd[H][l]);
          Yo[vsw<NP>(base + H * step)] = B.sum<3>();
        }
      }
    }
    __syncthreads();
    ok = cold == 0;
  }
  if (!ok) {
    double* const Yd = reinterpret_cast<double*>(Y);
    lift_lines_fp64<NP, NT>(Pe, D, Yd + 12 * n3, Yd);
    lift_nodes_fp64<NP, NT>(Me, Yd);
  }
  // ---- node by node: sJ M digits (< 2^58), the gradients with 2 bits below the digits' unit, and their traces
  // (one scale for each component of the gradient: in a flat element that of the flat direction meets the large
  // metric terms, the others the small ones)
  int sM[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) sM[d] = ok ? 59 - ((int)floorf(ml[14 + d]) + 1) : 0;
#pragma unroll 1
  for (int it = 0; it < (ok ? NPT : 0); ++it) {
    const int node = tid + it * NT;
    if (node >= n3) break;
    double g[12];
    const double sj = Me[9 * n3 + node];
    const int ej = fx_exp(fx_mag(sj));
    const FxDig J = fd_from(sj, fx_r0(59 - ej));  // sj 2^(59-ej) in [2^58, 2^59)
    FxDig M[9];
#pragma unroll
    for (int c = 0; c < 9; ++c) {
      FxDot p;
      p.add(fd_from(Me[c * n3 + node], fx_r0(sM[c % 3])), J);
      M[c] = fd_split(p.sum());
    }
    const int sn = vsw<NP>(node);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      FxDig y[3];
#pragma unroll
      for (int dir = 0; dir < 3; ++dir) y[dir] = fd_split(Y[(dir * 4 + v) * n3 + sn]);
      // g = r 2^(k - sM): scales of sJ M, of y, of the product
      const int k = -((59 - ej - 60) + (57 - fx_exp(mag[v]) + lb.sD - 60 + 3) - 60 + 2);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        FxDot p;
#pragma unroll
        for (int dir = 0; dir < 3; ++dir) p.add(y[dir], M[3 * dir + d]);
        g[d * 4 + v] = fx_scaled(p.sum<2>(), k - sM[d]);
      }
    }
    if constexpr (EXACT) {
      put_gradients<NP>(g, node, (size_t)e, es, nSides, Gvol, Gf);
    } else {
      // this node's derivatives are read: its gradients take their place
#pragma unroll
      for (int c = 0; c < 12; ++c) Y[c * n3 + vsw<NP>(node)] = __double_as_longlong(g[c]);
    }
  }
  if (!EXACT || !ok) {
    __syncthreads();
    // surface part, one thread per face node, one normal direction per pass (its two faces share no node)
#pragma unroll 1
    for (int dir = 0; dir < 3; ++dir) {
      for (int t = tid; t < 2 * n2; t += NT) {
        const bool minus = t < n2;
        const int ab = minus ? t : t - n2, a = ab % n, b = ab / n;
        const int ls = dir == 0 ? (minus ? L_XI_MINUS : L_XI_PLUS)
                                : (dir == 1 ? (minus ? L_ETA_MINUS : L_ETA_PLUS) : (minus ? L_ZETA_MINUS : L_ZETA_PLUS));
        const int node = face_node(n, ls, a, b, minus ? 0 : N);
        const int side = es[2 * (ls - 1)], flip = es[2 * (ls - 1) + 1];
        int p, q;
        s2v2_inv(N, a, b, flip, ls, p, q);
        const double* pm = Pf + (size_t)side * 6 * n2 + p + n * q;
        const double* ps = pm + (size_t)nSides * 6 * n2;
        const double* fg = Fgeo + (size_t)side * 10 * n2 + p + n * q;
        const double w = Lhat * 0.5 * fg[9 * n2] * Me[9 * n3 + node];
        const double nv[3] = {w * fg[0], w * fg[n2], w * fg[2 * n2]};
        double* const Gs = reinterpret_cast<double*>(Y) + vsw<NP>(node);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const double fl = ps[liftc(v) * n2] - pm[liftc(v) * n2];
#pragma unroll
          for (int d = 0; d < 3; ++d) Gs[(d * 4 + v) * n3] = Gs[(d * 4 + v) * n3] + fl * nv[d];
        }
      }
      __syncthreads();
    }
#pragma unroll 1
    for (int node = tid; node < n3; node += NT) {
      double g[12];
#pragma unroll
      for (int c = 0; c < 12; ++c) g[c] = reinterpret_cast<const double*>(Y)[c * n3 + vsw<NP>(node)];
      put_gradients<NP>(g, node, (size_t)e, es, nSides, Gvol, Gf);
    }
  }
}

}  // namespace gx

// k_volume_wfx: the volume kernel of the FP64 form for the weak form, on Gauss and Gauss-Lobatto nodes, in block
// fixed-point arithmetic on the integer pipes (dg_fx.cuh).
//
// VolInt_weakForm (src/dg/volint.f90:129-188) with EvalTransformedEulerFlux3D_fast (flux.f90:137-186) and
// EvalTransformedDiffFlux3D (:619-697), ApplyDMatrix (applydmatrix.t90:19-75), SurfIntCons (surfint.t90:352-586),
// -1, the Jacobian and the LSERK-W2 stage.  k_volume spends 240 FP64 instructions per node on this (N = 5,
// Navier-Stokes; 65 cycles each per warp and sub-partition); here the fluxes and the contractions are integer
// products and FP64 is left to the viscous stresses, (E + p)/rho, the five conversions, the Jacobian and the
// stage update.
//
// One element per block.  Node by node the contravariant fluxes go into shared memory as integers with one scale
// for each kind of row (mass, momentum, energy) over the three directions; then one thread per line and row
// contracts the line with D_hat in even and odd parts (it is centro-antisymmetric), adds the line's two face
// fluxes with their L_hat the same way, and puts the results in the fluxes' place; the three directions' results
// of a node are integers of one scale and are added up exactly.  24^3 curved, N = 5, Gauss, Navier-Stokes: 1.29 ms
// before, 0.905 ms; 48^3 Euler, N = 3: 1.84 and 1.19 ms.  With one scale for all rows and directions 0.87 and
// 1.04 ms, but on flat elements (1:100) the errors of the smallest row grew to 95 times the FP64 kernel's.
#pragma once
#include "dg_fx.cuh"
#include "dg_kernels.cuh"
#include "dg_volume_fx.cuh"

namespace gx {

template <int NP> struct VolWfx {
  static constexpr int n3 = NP * NP * NP, work = n3 > 5 * NP * NP ? n3 : 5 * NP * NP;
  // (n = 10: shared memory holds one block per SM; 12^3, Gauss, Navier-Stokes 0.667 ms with 256 threads, 0.551 with 512)
  static constexpr int NT = NP == 10 ? 512 : (work >= 256 ? 256 : (work + 31) / 32 * 32);
  static constexpr int MINB = 640 / NT > 16 ? 16 : 640 / NT;  // 96 registers per thread
  static constexpr size_t smem = sizeof(fx64) * 15 * n3;
};
// D_hat, and L_hat of the plus and minus faces, in even and odd parts, limbs times 2^sD (|.| < 2^60):
//   A = sum even(i,l) (f_l + f_(N-l)) + lo(i) (F_plus - F_minus),  B = sum odd(i,l) (f_l - f_(N-l)) + le(i) (F_plus + F_minus)
//   y(i) = A + B,  y(N-i) = B - A  (odd n: the middle node is the last column of even and the last row of odd)
template <int NP> struct VolWfxBasis {
  static constexpr int H = NP / 2, HE = (NP + 1) / 2;
  FxLimb even[H][HE], odd[HE][H], lo[H], le[HE];
  int sD, S;  // S: shift of the contractions, 3 * 2^59 * (largest row sum of |D_hat|, |L_hat|) * 2^(sD - 64 + S) < 2^63
};
// one direction: metric terms * 2^sM, left shifts of the products, right shifts of M.m, scales of the rows' fluxes;
// the stresses' scales
struct VolWfxDir {
  int sM, hV, hG[3], hE, k0, km, kE, t[5];
};
struct VolWfxScale {
  VolWfxDir d[3];
  int s_m, s_v, s_p, s_E, s_t, s_q, t[5], ok;
};
// largest magnitudes: W_M2, W_U2 float bits of |m|^2 and |u|^2; W_R: 1/rho; W_F: face fluxes [direction][row]
enum { W_M2, W_U2, W_P, W_E, W_TAU, W_TQ, W_F, W_V = W_F + 15, W_R, W_NMAX, W_PMIN = W_NMAX, W_RMIN, W_N };

// Scales of one element, by the first warp (lanes 0-2: one direction each).  Rows, with Mm = M_d.m (m = rho u): mass
// Mm, momentum c: Mm v_c + M_d,c p - M_d.tau_c, energy Mm (E+p)/rho - M_d.tq; each below 2^59 at its scale 2^t, the
// face fluxes too, so that the mixed products of a line's contraction (limbs of |D_hat| < 2^60, at most five products
// of sums of two and one face term) stay below 2^63; the contraction is shifted by as much as the rows of D_hat and
// L_hat allow (VolWfxBasis::S), so that the sum of three directions stays below 2^63.
// p, the stresses and (E+p)/rho have one scale each for the three directions, and the products of a direction's
// row are shifted to it at the end; Mm is shifted to the scale of M p before its product with v.
// Elements whose densities differ by more than 2^3 to 2^4 take the FP64 sums: at one pressure and velocity, rho u and
// (E+p)/rho have their maxima at opposite nodes, and the energy row's bound is above its products by the contrast
// (errors of the worst row, contrasts 8, 16, 64, 256: 0.65, 1.2, 2.4 and 5 times the FP64 kernel's).  So do flat
// elements, from 10:1 on here (8:1, 16:1, 64:1 and 256:1 at N = 2: 0.9, 1.1, 3.9 and 13 times), and those whose stresses exceed
// the pressure as there (vol_fx_scales; 4 to 6 times).
template <int PARAB>
__device__ __forceinline__ void vol_wfx_scales(const unsigned* mag, const float* MetL, VolWfxScale& S, int lane) {
  const int d = min(lane, 2);
  bool ok = MetL[d] < 200.f;
  for (int c = 0; c < W_NMAX; ++c)
    ok = ok && (c <= W_U2 ? mag[c] < 0x7b000000u : mag[c] < ((c < W_TAU ? 1022u + 150u : 1022u + 600u) << 20));
  const unsigned lowest = (1022u - 150u) << 20;
  ok = ok && (mag[W_V] == 0u || mag[W_V] >= (1023u - 60u) << 20);  // the range of fx_float
  ok = ok && mag[W_PMIN] > lowest && mag[W_E] > lowest && (mag[W_P] >> 20) - (mag[W_PMIN] >> 20) <= 8;
  ok = ok && mag[W_RMIN] > lowest && (mag[W_R] >> 20) - (mag[W_RMIN] >> 20) <= 3;
  const float LM = ok ? MetL[d] : 0.f;
  const float Lm = 0.5f * __log2f(__uint_as_float(mag[W_M2])) + 1e-4f, Lu = 0.5f * __log2f(__uint_as_float(mag[W_U2])) + 1e-4f;
  const float Lp = fx_log2(mag[W_P]), LE = fx_log2(mag[W_E]);
  const float Lt = fx_log2(mag[W_TAU]) + 0.8f, Lq = fx_log2(mag[W_TQ]) + 0.8f;
  const float LV = LM + Lm;
  ok = ok && fx_flatness(MetL) <= 3.25f && (!PARAB || Lt <= Lp + 2.8f);
  VolWfxDir o;
  o.sM = 59 - ((int)floorf(LM) + 1);
  const int s_m = 59 - ((int)floorf(Lm) + 1), s_v = 59 - ((int)floorf(Lu) + 1);
  const int sV = (int)floorf(60.4f - LV);
  o.hV = sV - (o.sM + s_m - 64);
  o.t[0] = (int)floorf(58.9f - fmaxf(LV, fx_log2(mag[W_F + 5 * d])));
  o.k0 = min(sV - o.t[0], 63);
  // scales of the momentum and energy rows
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    float L = fx_lse(LV + Lu, (ok ? MetL[3 + 3 * d + c] : 0.f) + Lp);
    if (PARAB) L = fx_lse(L, LM + Lt);
    o.t[1 + c] = (int)floorf(58.9f - fmaxf(L, fx_log2(mag[W_F + 5 * d + 1 + c])));
  }
  float Le = LV + LE;
  if (PARAB) Le = fx_lse(Le, LM + Lq);
  o.t[4] = (int)floorf(58.9f - fmaxf(Le, fx_log2(mag[W_F + 5 * d + 4])));
  // p and the stresses: below 2^60, M p no finer than Mm v can be, and not finer than the rows' scales; tq in the
  // same way beside Mm (E+p)/rho
  const int s_E = 60 - fx_exp(mag[W_E]);
  int s_p = min((int)floorf(PARAB ? fminf(59.9f - Lp, 59.9f - Lt) : 59.9f - Lp), sV + s_v - o.sM);
  s_p = min(s_p, min(o.t[1], min(o.t[2], o.t[3])) - o.sM + 63);
  int s_q = min(PARAB ? (int)floorf(59.9f - Lq) : 100000, min(sV + s_E, o.t[4] + 63) - o.sM);
#pragma unroll
  for (int x = 1; x < 4; x <<= 1) {
    s_p = min(s_p, __shfl_xor_sync(0xffffffffu, s_p, x));
    s_q = min(s_q, __shfl_xor_sync(0xffffffffu, s_q, x));
  }
  o.km = min(sV + s_v - o.sM - s_p, 63);
  o.kE = min(sV + s_E - o.sM - s_q, 63);
  auto in = [](int h) { return h >= 1 && h <= 31; };
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    o.t[1 + c] = min(o.t[1 + c], o.sM + s_p - 64 + 31);
    o.hG[c] = o.t[1 + c] - (o.sM + s_p - 64);
    ok = ok && in(o.hG[c]);
  }
  o.t[4] = min(o.t[4], o.sM + s_q - 64 + 31);
  o.hE = o.t[4] - (o.sM + s_q - 64);
  ok = ok && in(o.hV) && in(o.hE) && o.k0 >= 0 && o.km >= 0 && o.kE >= 0;
  ok = __all_sync(0xffffffffu, ok);
  int tr[5];
#pragma unroll
  for (int r = 0; r < 5; ++r) {
    tr[r] = o.t[r];
#pragma unroll
    for (int x = 1; x < 4; x <<= 1) tr[r] = min(tr[r], __shfl_xor_sync(0xffffffffu, tr[r], x));
  }
  if (lane < 3) S.d[d] = o;
  if (lane == 0) {
    S.s_m = s_m; S.s_v = s_v; S.s_p = s_p; S.s_E = s_E; S.s_t = s_p; S.s_q = s_q;
    for (int r = 0; r < 5; ++r) S.t[r] = tr[r];
    S.ok = ok;
  }
}

template <int NP, int PARAB>
__global__ void __launch_bounds__(VolWfx<NP>::NT, VolWfx<NP>::MINB)
k_volume_wfx(const double* __restrict__ U, const double* __restrict__ Pvol, const double* __restrict__ Gvol,
             const double* __restrict__ Met, const float* __restrict__ MetL, const double* __restrict__ Flux,
             const int* __restrict__ E2S, const __grid_constant__ VolWfxBasis<NP> wb, DevBasis<double> basis, int gauss,
             Gas<double> gas, RKArgs rk, int rkmode) {
  using C = VolWfx<NP>;
  constexpr int n = NP, n2 = NP * NP, n3 = NP * NP * NP, N = NP - 1, NT = C::NT;
  constexpr int H = VolWfxBasis<NP>::H, HE = VolWfxBasis<NP>::HE;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  fx64* const A = reinterpret_cast<fx64*>(smem_raw);  // [3][5][n3]
  __shared__ unsigned mag[W_N];
  __shared__ VolWfxScale sc;
  __shared__ int es[12];
  const int e = blockIdx.x, tid = threadIdx.x;
  if (tid < W_N) mag[tid] = tid < W_NMAX ? 0u : 0xffffffffu;
  if (tid < 12) es[tid] = E2S[(size_t)e * 12 + tid];
  __syncthreads();
  const double* const Pe = Pvol + (size_t)e * 7 * n3;
  const double* const Me = Met + (size_t)e * 10 * n3;
  const double* const Ue = U + (size_t)e * 5 * n3;
  const double* const Ge = PARAB ? Gvol + (size_t)e * 15 * n3 : nullptr;
  // ---- largest magnitudes; (E + p)/rho and the stresses wait in the node's slots as FP64
  {
    unsigned m[6] = {0u, 0u, 0u, 0u, 0u, 0u}, mV = 0u, pmin = 0xffffffffu, mr = 0u, rmin = 0xffffffffu;
    vol_flux_max<NP, NT>(Flux, es, &mag[W_F]);
#pragma unroll 1
    for (int node = tid; node < n3; node += NT) {
      const double* P = Pe + node;
      const double vel[3] = {P[n3], P[2 * n3], P[3 * n3]}, p = P[4 * n3];
      const double srho = P[6 * n3], Ep = (Ue[node * 5 + 4] + p) * srho;
      mr = max(mr, fx_mag(srho));
      rmin = min(rmin, fx_mag(srho));
      fx64* const a = A + vsw<NP>(node);
      a[0] = __double_as_longlong(Ep);
      auto norm2 = [](double x, double y, double z) {
        const float u = fx_float(fx_mag(x)), v = fx_float(fx_mag(y)), w = fx_float(fx_mag(z));
        return __float_as_uint(u * u + v * v + w * w);
      };
      const unsigned mm = max(fx_mag(Ue[node * 5 + 1]), max(fx_mag(Ue[node * 5 + 2]), fx_mag(Ue[node * 5 + 3])));
      const unsigned mv = max(fx_mag(vel[0]), max(fx_mag(vel[1]), fx_mag(vel[2])));
      mV = max(mV, min(mm, mv));
      m[W_M2] = max(m[W_M2], norm2(Ue[node * 5 + 1], Ue[node * 5 + 2], Ue[node * 5 + 3]));
      m[W_U2] = max(m[W_U2], norm2(vel[0], vel[1], vel[2]));
      m[W_P] = max(m[W_P], fx_mag(p));
      pmin = min(pmin, fx_mag(p));
      m[W_E] = max(m[W_E], fx_mag(Ep));
      if constexpr (PARAB) {
        const double* G = Ge + node;
        const double gx[5] = {0., G[n3], G[2 * n3], G[3 * n3], G[4 * n3]};
        const double gy[5] = {0., G[6 * n3], G[7 * n3], G[8 * n3], G[9 * n3]};
        const double gz[5] = {0., G[11 * n3], G[12 * n3], G[13 * n3], G[14 * n3]};
        double tau[6], tq[3];
        visc_stress(gx, gy, gz, vel, gas.mu, gas.lambda, tau, tq);
#pragma unroll
        for (int c = 0; c < 6; ++c) { m[W_TAU] = max(m[W_TAU], fx_mag(tau[c])); a[(1 + c) * n3] = __double_as_longlong(-tau[c]); }
#pragma unroll
        for (int c = 0; c < 3; ++c) { m[W_TQ] = max(m[W_TQ], fx_mag(tq[c])); a[(7 + c) * n3] = __double_as_longlong(-tq[c]); }
      }
    }
#pragma unroll
    for (int c = 0; c < (PARAB ? 6 : 4); ++c) fx_block_max(m[c], &mag[c]);
    fx_block_max(mV, &mag[W_V]);
    fx_block_min(pmin, &mag[W_PMIN]);
    fx_block_max(mr, &mag[W_R]);
    fx_block_min(rmin, &mag[W_RMIN]);
  }
  __syncthreads();
  if (tid < 32) vol_wfx_scales<PARAB>(mag, MetL + (size_t)e * kMetL, sc, tid);
  __syncthreads();
  if (sc.ok) {
    // ---- contravariant fluxes
    {
      const VolWfxScale& s = sc;
#pragma unroll 1
      for (int node = tid; node < n3; node += NT) {
        fx64* const a = A + vsw<NP>(node);
        auto raw = [&](int slot) { return __longlong_as_double(a[slot * n3]); };
        const FxLimb Ep = fx_limb(fx_from(raw(0), fx_r0(s.s_E)));
        FxLimb T[9];
        if constexpr (PARAB) {
#pragma unroll
          for (int c = 0; c < 6; ++c) T[c] = fx_limb(fx_from(raw(1 + c), fx_r0(s.s_t)));
#pragma unroll
          for (int c = 0; c < 3; ++c) T[6 + c] = fx_limb(fx_from(raw(7 + c), fx_r0(s.s_q)));
        }
        FxLimb mo[3], ve[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          mo[c] = fx_limb(fx_from(Ue[node * 5 + 1 + c], fx_r0(s.s_m)));
          ve[c] = fx_limb(fx_from(Pe[(1 + c) * n3 + node], fx_r0(s.s_v)));
        }
        const FxLimb p = fx_limb(fx_from(Pe[4 * n3 + node], fx_r0(s.s_p)));
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const VolWfxDir& sd = s.d[d];
          FxLimb M[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) M[c] = fx_limb(fx_from(Me[(3 * d + c) * n3 + node], fx_r0(sd.sM)));
          const fx64 Mm = fx_unbias64(fx_dot(M[0], mo[0], M[1], mo[1], M[2], mo[2], sd.hV), sd.hV);
          const FxLimb Mk = fx_limb(fx_sar(Mm, sd.km)), Ml = fx_limb(fx_sar(Mm, sd.kE));
          fx64* const o = a + d * 5 * n3;
          o[0] = fx_sar(Mm, sd.k0);
          const int tr[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            fx64 m = fx_mid(M[c], p, fx_mid(Mk, ve[c], kFxMid));
            if constexpr (PARAB) m = fx_mid(M[2], T[tr[c][2]], fx_mid(M[1], T[tr[c][1]], fx_mid(M[0], T[tr[c][0]], m)));
            fx64 t = fx_mad(M[c].h, p.h, fx_mad(Mk.h, ve[c].h, fx_up(m)));
            if constexpr (PARAB)
              t = fx_mad(M[2].h, T[tr[c][2]].h, fx_mad(M[1].h, T[tr[c][1]].h, fx_mad(M[0].h, T[tr[c][0]].h, t)));
            o[(1 + c) * n3] = fx_unbias64(fx_shift(t, m, sd.hG[c]), sd.hG[c]);
          }
          fx64 m = fx_mid(Ml, Ep, kFxMid);
          if constexpr (PARAB) m = fx_mid(M[2], T[8], fx_mid(M[1], T[7], fx_mid(M[0], T[6], m)));
          fx64 t = fx_mad(Ml.h, Ep.h, fx_up(m));
          if constexpr (PARAB) t = fx_mad(M[2].h, T[8].h, fx_mad(M[1].h, T[7].h, fx_mad(M[0].h, T[6].h, t)));
          o[4 * n3] = fx_unbias64(fx_shift(t, m, sd.hE), sd.hE);
        }
      }
    }
    __syncthreads();
    // ---- lines: one thread per direction, row and line
#pragma unroll 1
    for (int task = tid; task < 15 * n2; task += NT) {
      const int dv = task / n2, li = task - dv * n2, dir = dv / 5, v = dv - dir * 5;
      const int step = dir == 0 ? 1 : (dir == 1 ? n : n2);
      const int base = dir == 0 ? n * li : (dir == 1 ? (li % n) + n2 * (li / n) : li);
      fx64* const f = A + dv * n3;
      const int rF = fx_r0(sc.d[dir].t[v]);
      auto face = [&](int ls) {
        const int side = es[2 * (ls - 1)], flip = es[2 * (ls - 1) + 1];
        int p, q;
        s2v2_inv(N, li % n, li / n, flip, ls, p, q);
        const fx64 x = fx_from(Flux[((size_t)side * 5 + v) * n2 + p + n * q], rF);
        return flip == 0 ? x : -x;
      };
      const fx64 Fm = face(dir == 0 ? L_XI_MINUS : (dir == 1 ? L_ETA_MINUS : L_ZETA_MINUS));
      const fx64 Fp = face(dir == 0 ? L_XI_PLUS : (dir == 1 ? L_ETA_PLUS : L_ZETA_PLUS));
      const FxLimb fs = fx_limb(Fp + Fm), fd = fx_limb(Fp - Fm);
      FxLimb ev[HE], od[H];
#pragma unroll
      for (int l = 0; l < H; ++l) {
        const fx64 a = f[vsw<NP>(base + l * step)], b = f[vsw<NP>(base + (N - l) * step)];
        ev[l] = fx_limb(a + b);
        od[l] = fx_limb(a - b);
      }
      if constexpr (NP % 2) ev[H] = fx_limb(f[vsw<NP>(base + H * step)]);
#pragma unroll
      for (int i = 0; i < HE; ++i) {
        fx64 mB = fx_mid(fs, wb.le[i], 0), hB = fx_mad(fs.h, wb.le[i].h, 0);
#pragma unroll
        for (int l = 0; l < H; ++l) { mB = fx_mid(od[l], wb.odd[i][l], mB); hB = fx_mad(od[l].h, wb.odd[i][l].h, hB); }
        const fx64 B = fx_shift(hB + (mB >> 32), mB, wb.S);
        if (i < H) {
          fx64 mA = fx_mid(fd, wb.lo[i], 0), hA = fx_mad(fd.h, wb.lo[i].h, 0);
#pragma unroll
          for (int l = 0; l < HE; ++l) { mA = fx_mid(ev[l], wb.even[i][l], mA); hA = fx_mad(ev[l].h, wb.even[i][l].h, hA); }
          const fx64 a = fx_shift(hA + (mA >> 32), mA, wb.S);
          f[vsw<NP>(base + i * step)] = a + B;
          f[vsw<NP>(base + (N - i) * step)] = B - a;
        } else {
          f[vsw<NP>(base + i * step)] = B;
        }
      }
    }
    __syncthreads();
  } else {
    vol_block_fp64<NP, -1, PARAB, NT>(Ue, Pe, Ge, Me, Flux, es, basis, gauss, gas.mu, gas.lambda, nullptr,
                                      reinterpret_cast<double*>(smem_raw));
    __syncthreads();
  }
  // ---- the three directions' sum, -1, the Jacobian, output / LSERK-W2 stage
  auto put = [&](int t, double ut) {
    const size_t g = (size_t)e * n3 * 5 + t;
    if (rkmode == 0) {
      rk.Ut[g] = ut;
    } else {
      const double utmp = rk.Ut_tmp[g] * rk.mRKA + ut;
      rk.Ut_tmp[g] = utmp;
      rk.U[g] = rk.U[g] + utmp * rk.b_dt;
    }
  };
  if (!sc.ok) {
    for (int t = tid; t < 5 * n3; t += NT) put(t, __longlong_as_double(A[t]));
    return;
  }
#pragma unroll 1
  for (int node = tid; node < n3; node += NT) {
    double ut[5];
    const fx64* const a = A + vsw<NP>(node);
    const double c = -Me[9 * n3 + node];
    const int ch = __double2hiint(c), cl = __double2loint(c);
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      fx64 r = 0;
#pragma unroll
      for (int d = 0; d < 3; ++d) r += fx_sar(a[(5 * d + v) * n3], min(sc.d[d].t[v] - sc.t[v], 63));
      const int k = sc.t[v] + wb.sD - 64 + wb.S;
      ut[v] = __ll2double_rn(r) * __hiloint2double(ch - (k << 20), cl);
    }
    if constexpr (NP <= 5) {
      // into the node's own slots
#pragma unroll
      for (int v = 0; v < 5; ++v) A[v * n3 + vsw<NP>(node)] = __double_as_longlong(ut[v]);
    } else {
#pragma unroll
      for (int v = 0; v < 5; ++v) put(node * 5 + v, ut[v]);
    }
  }
  if constexpr (NP <= 5) {
    // out in the order of the state's memory: a step of 8^3 elements at N = 3 takes 154 against 164 us; from N = 5 on
    // the kernel is 1 to 2% slower that way
    __syncthreads();
#pragma unroll 2
    for (int t = tid; t < 5 * n3; t += NT) put(t, __longlong_as_double(A[(t % 5) * n3 + vsw<NP>(t / 5)]));
  }
}

}  // namespace gx

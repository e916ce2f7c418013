// k_volume_fx: the volume kernel of the FP64 form on Gauss-Lobatto nodes for the split forms PI and KG,
// in block fixed-point arithmetic on the integer pipes (dg_fx.cuh).
//
// VolInt_splitForm (src/dg/volint.f90:211-353), the viscous volume integral (EvalTransformedDiffFlux3D,
// flux.f90:619-697, with D_hat^T), SurfIntCons (surfint.t90:352-586), -1, the Jacobian and the LSERK-W2
// stage (vector.f90:163-183).  What k_volume computes with 518 FP64 instructions per node (N=7) takes 47
// here (viscous stresses, the Jacobian, the stage update); the rest runs on the integer pipes.
//
// Summation by parts on Gauss-Lobatto nodes brings every term of a line to one antisymmetric form.  With
// Q(i,l) = w_i DVolSurf(l,i) (i != l), Q(i,l) = -Q(l,i):
//   split form    w_i sum_l DVolSurf(l,i) F#(i,l)   = sum_l Q(i,l) F#(i,l)
//   viscous part  w_i sum_l D_hat^T(l,i) f(l)       = sum_l Q(i,l) (f(i) + f(l))
//   surface       w_i L_hat(i) F                    = F on the line's end nodes
// so a pair's flux is formed once, G = Q(a,b) (F#(a,b) + f(a) + f(b)), added to node a and subtracted
// from node b, and the face fluxes are added to the end nodes as they are; 1/w_i is applied at the end.
//
// Mapping: one element per block.  A warp holds whole lines of one direction.  For even n a thread owns the
// nodes k and k + n/2 of its line (k < n/2): their own pair first, then the pairs with the thread s places
// on, s = 1 .. (n/2-1)/2 (four pairs from two partner nodes), and for even n/2 two of the four pairs with the
// thread n/4 places on, whose thread evaluates the other two: n-1 pairs per thread, each of the line's
// n(n-1)/2 pairs once.  For odd n a thread owns one node and evaluates the pairs (i, i+d mod n),
// d = 1 .. (n-1)/2.  A pair's G stays with its thread for the own node and reaches the partner's thread by
// warp shuffles.  Against one thread per line this needs the accumulators of two nodes instead of n, and
// against one node per thread half of the shared-memory reads.
#pragma once
#include "dg_fx.cuh"
#include "dg_kernels.cuh"

namespace gx {

template <int NP> struct VolFx {
  static constexpr int OWN = NP % 2 ? 1 : 2;                      // nodes of a line per thread
  static constexpr int TPL = NP / OWN;                            // threads per line
  static constexpr int LPW = 32 / TPL;                            // lines per warp
  static constexpr int TPD = (NP * NP + LPW - 1) / LPW;           // warp tasks per direction
  static constexpr int TPW = (OWN == 1 && TPD > 1) || TPD > 16 ? 2 : 1;         // tasks of one warp per direction
  // warps and threads of a block (n = 10: one warp more, so that vol_block_fp64's 300 lines have a thread each)
  static constexpr int NW = NP == 10 ? 10 : (TPD + TPW - 1) / TPW, NT = 32 * NW;
  static constexpr int NPT = (NP * NP * NP + NT - 1) / NT;        // nodes per thread
  // blocks per SM for 128 registers per thread (512 threads), where shared memory holds them
  static constexpr int MINB = NP >= 9 ? 1 : (512 / NT < 16 ? 512 / NT : 16);
  // shared-memory slots of n^3 words: rho, aux, u, v, w, p, then per direction the metric terms (3) and
  // the viscous fluxes (4), overwritten by the direction's five sums
  __host__ __device__ static constexpr int dslots(int parab) { return parab ? 7 : 5; }
  __host__ __device__ static constexpr size_t smem(int parab) {
    return sizeof(fx64) * (size_t)(6 + 3 * dslots(parab)) * NP * NP * NP;
  }
};
// what the kernel needs of the basis: limbs of Q(i,l) 2^62 at [l + n i] and of w_0/w_i 2^60
template <int NP> struct VolFxBasis {
  FxLimb Q[NP * NP], iw[NP];
};
// MetL[e][kMetL]: log2 of the largest |M_d| (2-norm; 3) of the element, of its largest |M_d,c| (9), SurfElem and |sJ|
// (one each), of the largest |M_d,c| and |SurfElem n_c| over directions and faces (3), or kFxNoScale where its geometry is outside the range the scales are made for (2^-150 .. 2^150); such
// elements take the FP64 path
constexpr int kMetL = 17;
constexpr float kFxNoScale = 1e9f;

// shifts of one direction (see vol_fx_scales) and the scales of its five rows
struct VolFxShift {
  int hV, hq, hg, hp, hG[3], hE;  // left shifts of the products
  int k0, km, kv;              // right shifts: g for the mass row, g for the momentum rows, V for KG's energy row
  int St, kt, Sq, kq;          // viscous fluxes: shift of the product, then right shift (momentum, energy rows)
  int sM, t[5];                // metric terms * 2^sM; sums * 2^t
};
struct VolFxScale {
  VolFxShift d[3];
  int s_rho, s_aux, s_p, s_vel, s_tau, s_tq, t[5], ok;
};
// largest magnitudes of the element: fx_mag words; X_U2: float bits of |u|^2; X_F: face fluxes [direction][row]
enum { X_RHO, X_AUX, X_U2, X_P, X_TAU, X_TQ, X_F, X_V = X_F + 15, X_NMAX,
       X_RHOMIN = X_NMAX, X_PMIN, X_N };

__device__ __forceinline__ float fx_lse(float a, float b) {
  const float m = fmaxf(a, b);
  return m + __log2f(exp2f(a - m) + exp2f(b - m));
}
// The scales of one element, by the first warp (lanes 0-2: one direction each).  L.. are log2 of bounds.
// A pair's terms, in units of 8 Q F# (density row: 4 Q F#):  V = Ms.us, q = rho_s V, g = Q q;
//   mass g;  momentum g us + 4 Q ps Ms + 8 Q fs;  energy g aux_s (+ 2 Q ps V for KG) + 8 Q fs.
// Products are shifted to use the range up: V, q < 2^61.4, g and the rows' sums of terms < 2^60.4, so that a
// node's sum over its partners (sum |Q| <= 3.92 for N <= 9, |Q| < 1) and its face flux (< 2^61) stay below
// 2^63.  Smaller contributions are shifted right to the scale that the largest allows.  The momentum rows c of a
// direction differ in their pressure term p M_d,c (flat elements: a direction's large metric terms meet p in one
// row only), so each row has its own last shift.
// What a row loses is the distance from its own terms to the element's largest, so elements where that can be more
// than the eight bits that the range has over FP64 take the FP64 sums: densities or pressures that differ by 2^8,
// elements flatter than about 19:1 (their |M_d||u| stands against M_d.u of the flat direction; errors of the worst
// row at 16:1, 64:1 and 256:1 at N = 2: 0.9, 2.4 and 10 times the FP64 kernel's), viscous stresses above four times
// the pressure (there a momentum row with a small velocity has nothing of the size of the largest one's terms:
// up to 2 times).  rho |u|^2 above the pressure costs nothing: the pressure itself, a difference of energies, has
// the round-off of the larger.
template <int SPLIT, int PARAB>
__device__ __forceinline__ void vol_fx_scales(const unsigned* mag, const float* MetL, VolFxScale& S, int lane) {
  const int d = min(lane, 2);
  bool ok = MetL[d] < 200.f;
  for (int c = 0; c < X_NMAX; ++c) ok = ok && (c == X_U2 || mag[c] < ((c < X_TAU ? 1022u + 150u : 1022u + 600u) << 20));
  const unsigned lowest = (1022u - 150u) << 20;
  ok = ok && mag[X_RHOMIN] > lowest && mag[X_PMIN] > lowest && mag[X_AUX] > lowest && mag[X_U2] < 0x7b000000u;
  ok = ok && (mag[X_V] == 0u || mag[X_V] >= (1023u - 60u) << 20);  // the range of fx_float
  ok = ok && (mag[X_RHO] >> 20) - (mag[X_RHOMIN] >> 20) <= 8 && (mag[X_P] >> 20) - (mag[X_PMIN] >> 20) <= 8;
  const float Lr = fx_log2(mag[X_RHO]), La = fx_log2(mag[X_AUX]), Lp = fx_log2(mag[X_P]);
  const float Lu = 0.5f * __log2f(__uint_as_float(mag[X_U2])) + 1e-4f, LM = ok ? MetL[d] : 0.f;
  const float Lt = fx_log2(mag[X_TAU]) + 0.8f, Lq = fx_log2(mag[X_TQ]) + 0.8f;
  ok = ok && fx_flatness(MetL) <= 4.25f && (!PARAB || Lt <= Lp + 2.8f);
  const int ev = (int)floorf(Lu) + 1, eM = (int)floorf(LM) + 1;
  const int s_rho = 61 - fx_exp(mag[X_RHO]), s_vel = 59 - ev, sM = 59 - eM;
  const int s_tau = 59 - fx_exp(mag[X_TAU]), s_tq = 59 - fx_exp(mag[X_TQ]);
  VolFxShift o;
  o.sM = sM;
  const float LV = 2.f + LM + Lu, Lqq = 1.f + Lr + LV;
  o.hV = (int)floorf(61.4f - LV) - (sM + s_vel - 64);
  const int sV = sM + s_vel - 64 + o.hV;
  o.hq = (int)floorf(61.4f - Lqq) - (s_rho + sV - 64);
  const int sq = s_rho + sV - 64 + o.hq;
  const int sg = (int)floorf(60.4f - Lqq);
  o.hg = sg - (sq - 2);
  // momentum rows
  int tm[3], tlow = 100000;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    float Lm = fx_lse(Lqq + 1.f + Lu, 4.f + Lp + (ok ? MetL[3 + 3 * d + c] : 0.f));
    if (PARAB) Lm = fx_lse(Lm, 4.f + LM + Lt);
    tm[c] = (int)floorf(fminf(60.4f - Lm, 58.f - fx_log2(mag[X_F + 5 * d + 1 + c])));
    tlow = min(tlow, tm[c]);
  }
  const int spx = (int)floorf(59.9f - Lp);
  // the shift of the row with the smallest scale; the others' are larger by their difference
  const int hl = max(2, max(tlow - (sg + s_vel - 64), tlow + 2 - (spx + sM - 64)));
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    tm[c] = min(tm[c], tlow + 31 - hl);
    o.hG[c] = hl + tm[c] - tlow;
  }
  o.km = min(sg + s_vel - 64 + hl - tlow, 63);
  const int sp = tlow + 2 - (sM - 64) - hl;
  // energy row
  float Le = Lqq + 1.f + La;
  if (SPLIT == DG_SPLIT_KG) Le = fx_lse(Le, 2.f + Lp + LV);
  if (PARAB) Le = fx_lse(Le, 4.f + LM + Lq);
  const int t4 = (int)floorf(fminf(60.4f - Le, 58.f - fx_log2(mag[X_F + 5 * d + 4])));
  const int he = SPLIT == DG_SPLIT_KG ? max(2, t4 + 65 - sp - sV) : 2;
  // p and aux have one scale for the three directions
  int s_p = min(61 - fx_exp(mag[X_P]), sp + 1), s_aux = min(61 - fx_exp(mag[X_AUX]), t4 - sg + 64 - he);
#pragma unroll
  for (int x = 1; x < 4; x <<= 1) {
    s_p = min(s_p, __shfl_xor_sync(0xffffffffu, s_p, x));
    s_aux = min(s_aux, __shfl_xor_sync(0xffffffffu, s_aux, x));
  }
  o.hp = sp + 2 - s_p;
  o.hE = t4 - sg - s_aux + 64;
  o.kv = SPLIT == DG_SPLIT_KG ? min(sp + sV - 64 + o.hE - t4 - 1, 63) : 0;
  // viscous fluxes: 8 Q f at the rows' scales, from M tau / 2^64 and M tq / 2^64
  const int ft = tlow + 5 - hl - (sM + s_tau - 64), fq = t4 + 5 - o.hE - (sM + s_tq - 64);
  o.St = max(1, ft); o.kt = min(o.St - ft, 63);
  o.Sq = max(1, fq); o.kq = min(o.Sq - fq, 63);
  // mass row
  const int t0 = (int)floorf(fminf((float)sg, 59.f - fx_log2(mag[X_F + 5 * d])));
  o.k0 = min(sg - t0, 63);
  o.t[0] = t0; o.t[1] = tm[0]; o.t[2] = tm[1]; o.t[3] = tm[2]; o.t[4] = t4;
  auto in = [](int h) { return h >= 1 && h <= 31; };
  ok = ok && in(o.hV) && in(o.hq) && in(o.hg) && in(o.hp) && in(o.hG[0]) && in(o.hG[1]) && in(o.hG[2]) && in(o.hE) && o.km >= 0 && o.k0 >= 0 && o.kv >= 0;
  if (PARAB) ok = ok && in(o.St) && in(o.Sq);
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
    S.s_rho = s_rho; S.s_aux = s_aux; S.s_p = s_p; S.s_vel = s_vel; S.s_tau = s_tau; S.s_tq = s_tq;
    for (int r = 0; r < 5; ++r) S.t[r] = tr[r];
    S.ok = ok;
  }
}
// largest magnitudes of an element's face fluxes into out[5 * direction + row].  Large blocks: a warp takes whole
// groups, one reduction each (24^3, N = 7: the kernel 1.86 ms, 1.88 with every warp in all 15 reductions).  Small
// blocks: all warps together, five loads in flight (64^3, N = 2, when it was written: 1.94 against 2.46 ms).
template <int NP, int NT>
__device__ __forceinline__ void vol_flux_max(const double* Flux, const int* es, unsigned* out) {
  constexpr int n2 = NP * NP, NW = NT / 32;
  auto minus = [](int dir) { return dir == 0 ? L_XI_MINUS : (dir == 1 ? L_ETA_MINUS : L_ZETA_MINUS); };
  auto plus = [](int dir) { return dir == 0 ? L_XI_PLUS : (dir == 1 ? L_ETA_PLUS : L_ZETA_PLUS); };
  if constexpr (NP >= 6) {
    const int lane = threadIdx.x & 31;
#pragma unroll 4
    for (int g = threadIdx.x >> 5; g < 15; g += NW) {
      const int dir = g / 5, v = g - 5 * dir;
      const double* const fm = Flux + ((size_t)es[2 * (minus(dir) - 1)] * 5 + v) * n2;
      const double* const fp = Flux + ((size_t)es[2 * (plus(dir) - 1)] * 5 + v) * n2;
      unsigned m = 0u;
#pragma unroll
      for (int t = 0; t < n2; t += 32)
        if (t + lane < n2) m = max(m, max(fx_mag(fm[t + lane]), fx_mag(fp[t + lane])));
      m = __reduce_max_sync(0xffffffffu, m);
      if (lane == 0) out[g] = m;
    }
  } else {
#pragma unroll 1
    for (int dir = 0; dir < 3; ++dir) {
      unsigned f[5] = {0u, 0u, 0u, 0u, 0u};
      for (int t = threadIdx.x; t < 2 * n2; t += NT) {
        const int ls = t < n2 ? minus(dir) : plus(dir);
        const double* fx = Flux + (size_t)es[2 * (ls - 1)] * 5 * n2 + (t < n2 ? t : t - n2);
#pragma unroll
        for (int v = 0; v < 5; ++v) f[v] = max(f[v], fx_mag(fx[v * n2]));
      }
#pragma unroll
      for (int v = 0; v < 5; ++v) fx_block_max(f[v], out + 5 * dir + v);
    }
  }
}

// The same sums in FP64 by the block, in the operations of k_volume: for elements whose values do not fit one scale
// per quantity (infinities and NaN, magnitudes outside 2^+-150, densities or pressures that differ by more than the
// scales allow within the element, which one scale would hold less exactly than FP64).  Bound by the FP64 pipe like
// k_volume, whose work it does: the viscous or weak fluxes once per node, each pair once (N = 7, 16^3, Navier-Stokes,
// all elements: 2.13 ms, k_volume 1.95; weak form on Gauss nodes 1.17 and 0.98; node by node from global memory they
// took 6.95 and 5.68).  SPLIT < 0: weak form.
// A: the block's shared memory, of which the fixed-point values are not needed any more (SPLIT < 0: 15 slots, else
// 27, or 21 for the Euler equations); the results are left there as [node][5].  D: n^2 words for the split form's
// matrix (the limbs' place: with words of its own the block of n = 4 fits an SM 14 instead of 15 times).
template <int NP, int SPLIT, int PARAB, int NT>
__device__ __noinline__ void vol_block_fp64(const double* U, const double* Pe, const double* Ge, const double* Me,
                                            const double* Flux, const int* es, DevBasis<double> basis, int gauss,
                                            double mu, double lambda, double* D, double* A) {
  constexpr int n = NP, n2 = NP * NP, n3 = NP * NP * NP, N = NP - 1, NPT = (n3 + NT - 1) / NT;
  constexpr int v0 = SPLIT < 0 ? 0 : 1, nvs = 5 - v0;  // slots of flux (d, v): d nvs + v - v0
  const int tid = threadIdx.x;
  double acc[NPT][5];
#pragma unroll
  for (int it = 0; it < NPT; ++it)
#pragma unroll
    for (int v = 0; v < 5; ++v) acc[it][v] = 0.;
  __syncthreads();
  if constexpr (SPLIT < 0 || PARAB) {
#pragma unroll 1
    for (int node = tid; node < n3; node += NT) {
      const double* const P = Pe + node;
      const double vel[3] = {P[n3], P[2 * n3], P[3 * n3]};
      double tau[6] = {0., 0., 0., 0., 0., 0.}, tq[3] = {0., 0., 0.};
      if constexpr (PARAB) {
        const double* const G = Ge + node;
        const double gx[5] = {0., G[n3], G[2 * n3], G[3 * n3], G[4 * n3]};
        const double gy[5] = {0., G[6 * n3], G[7 * n3], G[8 * n3], G[9 * n3]};
        const double gz[5] = {0., G[11 * n3], G[12 * n3], G[13 * n3], G[14 * n3]};
        visc_stress(gx, gy, gz, vel, mu, lambda, tau, tq);
      }
      const double *const Un = U + node * 5, p = P[4 * n3], Ep = SPLIT < 0 ? (Un[4] + p) * P[6 * n3] : 0.;
      double* const a = A + vsw<NP>(node);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const double m0 = Me[3 * d * n3 + node], m1 = Me[(3 * d + 1) * n3 + node], m2 = Me[(3 * d + 2) * n3 + node];
        double f[5] = {0., 0., 0., 0., 0.};
        if constexpr (SPLIT < 0) {
          const double mm = m0 * Un[1] + m1 * Un[2] + m2 * Un[3];
          f[0] = mm;
          f[1] = mm * vel[0] + m0 * p;
          f[2] = mm * vel[1] + m1 * p;
          f[3] = mm * vel[2] + m2 * p;
          f[4] = mm * Ep;
        }
        if constexpr (PARAB) {
          f[1] = f[1] - m0 * tau[0] - m1 * tau[3] - m2 * tau[4];
          f[2] = f[2] - m0 * tau[3] - m1 * tau[1] - m2 * tau[5];
          f[3] = f[3] - m0 * tau[4] - m1 * tau[5] - m2 * tau[2];
          f[4] = f[4] - m0 * tq[0] - m1 * tq[1] - m2 * tq[2];
        }
#pragma unroll
        for (int v = v0; v < 5; ++v) a[(d * nvs + v - v0) * n3] = f[v];
      }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < NPT; ++it) {
      const int node = tid + it * NT;
      if (node >= n3) break;
      const int i = node % n, j = (node / n) % n, k = node / n2;
#pragma unroll 4
      for (int l = 0; l < n; ++l) {
        const double ci = basis.DhatT[l + n * i], cj = basis.DhatT[l + n * j], ck = basis.DhatT[l + n * k];
        const int ni = vsw<NP>(l + n * (j + n * k)), nj = vsw<NP>(i + n * (l + n * k)), nk = vsw<NP>(i + n * (j + n * l));
#pragma unroll
        for (int v = v0; v < 5; ++v)
          acc[it][v] = acc[it][v] + ci * A[(v - v0) * n3 + ni] + ck * A[(2 * nvs + v - v0) * n3 + nk] +
                       cj * A[(nvs + v - v0) * n3 + nj];
      }
    }
    __syncthreads();
  }
  if constexpr (SPLIT >= 0) {
    // one thread per line, node b's share of a pair (a, b) to the line's own sums in shared memory
    double* const S = A + (PARAB ? 12 : 6) * n3;  // [3][5][n3]
    for (int t = tid; t < n2; t += NT) D[t] = SPLIT == DG_SPLIT_PI ? dp_scale(basis.DVS[t], -3) : basis.DVS[t];
#pragma unroll 1
    for (int node = tid; node < n3; node += NT) {
      const double* const P = Pe + node;
      double* const a = A + vsw<NP>(node);
      const double rho = P[0], u = P[n3], v = P[2 * n3], w = P[3 * n3], p = P[4 * n3];
      a[0] = rho; a[2 * n3] = u; a[3 * n3] = v; a[4 * n3] = w; a[5 * n3] = SPLIT == DG_SPLIT_PI ? 4. * p : p;
      a[n3] = pair_aux<SPLIT, double>(rho, u, v, w, U[node * 5 + 4], p, P[6 * n3]);
      for (int c = 0; c < 15; ++c) S[c * n3 + vsw<NP>(node)] = 0.;
    }
    __syncthreads();
#pragma unroll 1
    for (int t = tid; t < 3 * n2; t += NT) {
      const int dir = t / n2, li = t - dir * n2, step = dir == 0 ? 1 : (dir == 1 ? n : n2);
      const int base = dir == 0 ? n * li : (dir == 1 ? (li % n) + n2 * (li / n) : li);
      double* const Sd = S + dir * 5 * n3;
      const double* const M = Me + 3 * dir * n3;
      auto load = [&](int s, PairNode<double>& x) {
        x.rho = A[s]; x.aux = A[n3 + s]; x.u = A[2 * n3 + s]; x.v = A[3 * n3 + s]; x.w = A[4 * n3 + s]; x.pm = A[5 * n3 + s];
        x.m1 = x.m2 = x.m3 = 0.;
      };
#pragma unroll 1
      for (int ia = 0; ia < n - 1; ++ia) {
        const int na = base + ia * step, sa = vsw<NP>(na);
        PairNode<double> a;
        load(sa, a);
        const double a0 = M[na], a1 = M[n3 + na], a2 = M[2 * n3 + na];
        double sum[5];
#pragma unroll
        for (int v = 0; v < 5; ++v) sum[v] = Sd[v * n3 + sa];
#pragma unroll 2
        for (int ib = ia + 1; ib < n; ++ib) {
          const int nb = base + ib * step, sb = vsw<NP>(nb);
          PairNode<double> b;
          load(sb, b);
          double F[5];
          const double M0 = a0 + M[nb], M1 = a1 + M[n3 + nb], M2 = a2 + M[2 * n3 + nb];
          if constexpr (SPLIT == DG_SPLIT_PI) {
            // 8 F, the density row 4 F, and DVolSurf / 8 (exact scalings)
            const double us = a.u + b.u, vs = a.v + b.v, ws = a.w + b.w, ps = a.pm + b.pm;
            const double q = (a.rho + b.rho) * (M0 * us + M1 * vs + M2 * ws);
            F[0] = q;
            F[1] = q * us + ps * M0;
            F[2] = q * vs + ps * M1;
            F[3] = q * ws + ps * M2;
            F[4] = q * (a.aux + b.aux);
          } else {
            split_pair_flux<SPLIT, double>(a, b, M0, M1, M2, 0., F);
          }
          const double dba = D[ib + n * ia], dab = D[ia + n * ib];
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            sum[v] = sum[v] + dba * F[v];
            Sd[v * n3 + sb] += dab * F[v];
          }
        }
#pragma unroll
        for (int v = 0; v < 5; ++v) Sd[v * n3 + sa] = sum[v];
      }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < NPT; ++it) {
      const int node = tid + it * NT, s = vsw<NP>(node);
      if (node < n3)
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          double x = S[v * n3 + s] + S[(5 + v) * n3 + s] + S[(10 + v) * n3 + s];
          if (SPLIT == DG_SPLIT_PI && v == 0) x = x * 2.;
          acc[it][v] = acc[it][v] + x;
        }
    }
    __syncthreads();
  }
  // the fluxes of the six faces (slave sides negated), then of each node's lines
#pragma unroll 1
  for (int t = tid; t < 6 * n2; t += NT) {
    const int ls = t / n2 + 1, ab = t - (ls - 1) * n2, side = es[2 * (ls - 1)], flip = es[2 * (ls - 1) + 1];
    int p, q;
    s2v2_inv(N, ab % n, ab / n, flip, ls, p, q);
    const double* const f = Flux + (size_t)side * 5 * n2 + p + n * q;
#pragma unroll
    for (int v = 0; v < 5; ++v) A[((ls - 1) * 5 + v) * n2 + ab] = flip == 0 ? f[v * n2] : -f[v * n2];
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < NPT; ++it) {
    const int node = tid + it * NT;
    if (node >= n3) break;
    const int i = node % n, j = (node / n) % n, k = node / n2;
    double ut[5] = {0., 0., 0., 0., 0.};
#pragma unroll 1
    for (int ls = 1; ls <= 6; ++ls) {
      const int dir = ls == L_XI_MINUS || ls == L_XI_PLUS ? 0 : (ls == L_ETA_MINUS || ls == L_ETA_PLUS ? 1 : 2);
      const int l = dir == 0 ? i : (dir == 1 ? j : k);
      if (!gauss && l != (is_minus(ls) ? 0 : N)) continue;
      const double Lh = is_minus(ls) ? basis.Lhm[l] : basis.Lhp[l];
      const double* const f = A + (ls - 1) * 5 * n2 + (dir == 0 ? j : i) + n * (dir == 2 ? j : k);
#pragma unroll
      for (int v = 0; v < 5; ++v) ut[v] = ut[v] + f[v * n2] * Lh;
    }
    const double sj = Me[9 * n3 + node];
#pragma unroll
    for (int v = 0; v < 5; ++v) acc[it][v] = (acc[it][v] + ut[v]) * -1. * sj;
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < NPT; ++it) {
    const int node = tid + it * NT;
    if (node < n3)
#pragma unroll
      for (int v = 0; v < 5; ++v) A[node * 5 + v] = acc[it][v];
  }
}

template <int NP, int SPLIT, int PARAB>
__global__ void __launch_bounds__(VolFx<NP>::NT, VolFx<NP>::MINB)
k_volume_fx(const double* __restrict__ U, const double* __restrict__ Pvol, const double* __restrict__ Gvol,
            const double* __restrict__ Met, const float* __restrict__ MetL, const double* __restrict__ Flux,
            const int* __restrict__ E2S, const VolFxBasis<NP>* __restrict__ fxb, DevBasis<double> basis, double iw0,
            Gas<double> gas, RKArgs rk, int rkmode) {
  using C = VolFx<NP>;
  constexpr int n = NP, n2 = NP * NP, n3 = NP * NP * NP, N = NP - 1, NT = C::NT, NPT = C::NPT, DS = C::dslots(PARAB);
  constexpr int OWN = C::OWN, TPL = C::TPL;
  constexpr int S_RHO = 0, S_AUX = 1, S_VEL = 2, S_P = 5;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  fx64* const A = reinterpret_cast<fx64*>(smem_raw);
  __shared__ __align__(8) VolFxBasis<NP> sb;
  __shared__ unsigned mag[X_N];
  __shared__ VolFxScale sc;
  __shared__ int es[12];
  const int e = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < X_N) mag[tid] = tid < X_NMAX ? 0u : 0xffffffffu;
  if (tid < 12) es[tid] = E2S[(size_t)e * 12 + tid];
  for (int t = tid; t < n2; t += NT) sb.Q[t] = fxb->Q[t];
  if (tid < n) sb.iw[tid] = fxb->iw[tid];
  __syncthreads();
  const double* const Pe = Pvol + (size_t)e * 7 * n3;
  const double* const Me = Met + (size_t)e * 10 * n3;
  const double* const Ue = U + (size_t)e * 5 * n3;
  const double* const Ge = PARAB ? Gvol + (size_t)e * 15 * n3 : nullptr;

  // ---- largest magnitudes of the element: node data, viscous stresses, face fluxes
  // (the values wait in the node's own shared-memory slots as FP64 for the scales: slots 0-5 the node data,
  // 6-14 the stresses)
  {
    vol_flux_max<NP, NT>(Flux, es, &mag[X_F]);
    unsigned m[6] = {0, 0, 0, 0, 0, 0}, mv = 0u, rmin = 0xffffffffu, pmin = 0xffffffffu;
#pragma unroll 1
    for (int node = tid; node < n3; node += NT) {
      const double* P = Pe + node;
      fx64* const a = A + vsw<NP>(node);
      const double rho = P[0], vel[3] = {P[n3], P[2 * n3], P[3 * n3]}, p = P[4 * n3];
      const double aux = pair_aux<SPLIT, double>(rho, vel[0], vel[1], vel[2], Ue[node * 5 + 4], p, P[6 * n3]);
      a[S_RHO * n3] = __double_as_longlong(rho);
      a[S_AUX * n3] = __double_as_longlong(aux);
      a[S_P * n3] = __double_as_longlong(p);
#pragma unroll
      for (int c = 0; c < 3; ++c) a[(S_VEL + c) * n3] = __double_as_longlong(vel[c]);
      m[X_RHO] = max(m[X_RHO], fx_mag(rho));
      rmin = min(rmin, fx_mag(rho));
      m[X_AUX] = max(m[X_AUX], fx_mag(aux));
      m[X_P] = max(m[X_P], fx_mag(p));
      pmin = min(pmin, fx_mag(p));
      const float u = fx_float(fx_mag(vel[0])), v = fx_float(fx_mag(vel[1])), w = fx_float(fx_mag(vel[2]));
      m[X_U2] = max(m[X_U2], __float_as_uint(u * u + v * v + w * w));
      mv = max(mv, max(fx_mag(vel[0]), max(fx_mag(vel[1]), fx_mag(vel[2]))));
      if constexpr (PARAB) {
        const double* G = Ge + node;
        const double gx[5] = {0., G[n3], G[2 * n3], G[3 * n3], G[4 * n3]};
        const double gy[5] = {0., G[6 * n3], G[7 * n3], G[8 * n3], G[9 * n3]};
        const double gz[5] = {0., G[11 * n3], G[12 * n3], G[13 * n3], G[14 * n3]};
        double tau[6], tq[3];
        visc_stress(gx, gy, gz, vel, gas.mu, gas.lambda, tau, tq);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          m[X_TAU] = max(m[X_TAU], fx_mag(tau[c]));
          a[(6 + c) * n3] = __double_as_longlong(tau[c]);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          m[X_TQ] = max(m[X_TQ], fx_mag(tq[c]));
          a[(12 + c) * n3] = __double_as_longlong(tq[c]);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < (PARAB ? 6 : 4); ++c) fx_block_max(m[c], &mag[c]);
    fx_block_max(mv, &mag[X_V]);
    fx_block_min(rmin, &mag[X_RHOMIN]);
    fx_block_min(pmin, &mag[X_PMIN]);
  }
  __syncthreads();
  if (warp == 0) vol_fx_scales<SPLIT, PARAB>(mag, MetL + (size_t)e * kMetL, sc, lane);
  __syncthreads();
  double* const Us = reinterpret_cast<double*>(smem_raw);  // Ut of the element, [node][5], at the end
  if (sc.ok) {
    // ---- node data to fixed point
    {
      const int r_rho = fx_r0(sc.s_rho), r_aux = fx_r0(sc.s_aux), r_vel = fx_r0(sc.s_vel), r_p = fx_r0(sc.s_p);
      const int r_tau = fx_r0(sc.s_tau), r_tq = fx_r0(sc.s_tq);
#pragma unroll 1
      for (int node = tid; node < n3; node += NT) {
        fx64* const a = A + vsw<NP>(node);
        auto raw = [&](int slot) { return __longlong_as_double(a[slot * n3]); };
        FxLimb T[9];
        if constexpr (PARAB) {
#pragma unroll
          for (int c = 0; c < 6; ++c) T[c] = fx_limb(fx_from(raw(6 + c), r_tau));
#pragma unroll
          for (int c = 0; c < 3; ++c) T[6 + c] = fx_limb(fx_from(raw(12 + c), r_tq));
        }
        a[S_RHO * n3] = fx_from(raw(S_RHO), r_rho);
        a[S_AUX * n3] = fx_from(raw(S_AUX), r_aux);
        a[S_P * n3] = fx_from(raw(S_P), r_p);
#pragma unroll
        for (int c = 0; c < 3; ++c) a[(S_VEL + c) * n3] = fx_from(raw(S_VEL + c), r_vel);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          fx64* const ad = a + (6 + d * DS) * n3;
          const int r_M = fx_r0(sc.d[d].sM);
          FxLimb M[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const fx64 x = fx_from(Me[(3 * d + c) * n3 + node], r_M);
            ad[c * n3] = x;
            M[c] = fx_limb(x);
          }
          if constexpr (PARAB) {
            // EvalTransformedDiffFlux3D: -M_d . (rows of tau), -M_d . tq
            const int St = sc.d[d].St, kt = sc.d[d].kt, Sq = sc.d[d].Sq, kq = sc.d[d].kq;
            auto row = [&](const FxLimb& a0, const FxLimb& a1, const FxLimb& a2, int S, int k) {
              return -fx_sar(fx_unbias64(fx_dot(M[0], a0, M[1], a1, M[2], a2, S), S), k);
            };
            ad[3 * n3] = row(T[0], T[3], T[4], St, kt);
            ad[4 * n3] = row(T[3], T[1], T[5], St, kt);
            ad[5 * n3] = row(T[4], T[5], T[2], St, kt);
            ad[6 * n3] = row(T[6], T[7], T[8], Sq, kq);
          }
        }
      }
    }
    __syncthreads();

    // ---- pairs, one direction after the other
    const int lsub = lane / TPL, pos = lane - lsub * TPL;
#pragma unroll 1
    for (int dir = 0; dir < 3; ++dir) {
      fx64* const Ad = A + (6 + dir * DS) * n3;
      const int step = dir == 0 ? 1 : (dir == 1 ? n : n2);
      const VolFxShift sh = sc.d[dir];
      fx64 acc[C::TPW][OWN][5];
      int so[C::TPW][OWN];
#pragma unroll
      for (int tw = 0; tw < C::TPW; ++tw) {
        // lanes without a line compute the element's last one again and store nothing
        const int li = min((warp + tw * C::NW) * C::LPW + lsub, n2 - 1);
        const int base = dir == 0 ? n * li : (dir == 1 ? (li % n) + n2 * (li / n) : li);
        // own nodes; the fixed-point data + 2^31 (see fx_sum)
        fx64 rho[OWN], aux[OWN], pm[OWN], vel[OWN][3], M[OWN][3];
#pragma unroll
        for (int o = 0; o < OWN; ++o) {
          const int s = vsw<NP>(base + (pos + o * TPL) * step);
          so[tw][o] = s;
          rho[o] = A[S_RHO * n3 + s] + kFxHalf;
          aux[o] = A[S_AUX * n3 + s] + kFxHalf;
          pm[o] = A[S_P * n3 + s] + kFxHalf;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            vel[o][c] = A[(S_VEL + c) * n3 + s] + kFxHalf;
            M[o][c] = Ad[c * n3 + s] + kFxHalf;
          }
#pragma unroll
          for (int c = 0; c < 5; ++c) acc[tw][o][c] = 0;
        }
        struct Node { fx64 rho, aux, pm, vel[3], M[3]; int s; };
        auto load = [&](int s, Node& b) {
          b.rho = A[S_RHO * n3 + s]; b.aux = A[S_AUX * n3 + s]; b.pm = A[S_P * n3 + s];
#pragma unroll
          for (int c = 0; c < 3; ++c) { b.vel[c] = A[(S_VEL + c) * n3 + s]; b.M[c] = Ad[c * n3 + s]; }
          b.s = s;
        };
        // Q times 8 x the pair's fluxes (the density row 4 x), each with the bias of its last product; the
        // bias cancels between the G a node adds and those it receives, except for the own pair
        auto pair = [&](int o, const Node& b, const FxLimb Q, fx64 (&G)[5]) {
          // the viscous fluxes of both nodes are read here: held as well, they would not leave enough registers
          auto fvs = [&](int c) { return fx_limb(Ad[(3 + c) * n3 + so[tw][o]] + Ad[(3 + c) * n3 + b.s]); };
          FxLimb us[3], Ms[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) { us[c] = fx_sum(vel[o][c], b.vel[c]); Ms[c] = fx_sum(M[o][c], b.M[c]); }
          const fx64 V = fx_dot(Ms[0], us[0], Ms[1], us[1], Ms[2], us[2], sh.hV);
          const FxLimb q = fx_unbias(fx_mul(fx_sum(rho[o], b.rho), fx_unbias(V, sh.hV), sh.hq), sh.hq);
          const fx64 g = fx_unbias64(fx_mul(Q, q, sh.hg), sh.hg);
          const FxLimb pq = fx_unbias(fx_mul(Q, fx_sum(pm[o], b.pm), sh.hp), sh.hp);
          const FxLimb gm = fx_limb(fx_sar(g, sh.km)), gl = fx_limb(g), as = fx_sum(aux[o], b.aux);
          G[0] = fx_sar(g, sh.k0);
          if constexpr (PARAB) {
#pragma unroll
            for (int c = 0; c < 3; ++c) G[1 + c] = fx_dot(gm, us[c], pq, Ms[c], Q, fvs(c), sh.hG[c]);
            const FxLimb f4 = fvs(3);
            if constexpr (SPLIT == DG_SPLIT_KG)
              G[4] = fx_dot(gl, as, pq, fx_limb(fx_sar(fx_unbias64(V, sh.hV), sh.kv)), Q, f4, sh.hE);
            else
              G[4] = fx_dot(gl, as, Q, f4, sh.hE);
          } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) G[1 + c] = fx_dot(gm, us[c], pq, Ms[c], sh.hG[c]);
            if constexpr (SPLIT == DG_SPLIT_KG)
              G[4] = fx_dot(gl, as, pq, fx_limb(fx_sar(fx_unbias64(V, sh.hV), sh.kv)), sh.hE);
            else
              G[4] = fx_mul(gl, as, sh.hE);
          }
        };
        auto get = [&](fx64 x, int from) { return (fx64)__shfl_sync(0xffffffffu, x, from); };
        if constexpr (OWN == 1) {
#pragma unroll
          for (int d = 1; d <= n / 2; ++d) {
            const int b = pos + d < n ? pos + d : pos + d - n;
            Node B;
            load(vsw<NP>(base + b * step), B);
            fx64 G[5];
            pair(0, B, sb.Q[b + n * pos], G);
            const int from = lane + (pos >= d ? -d : n - d);  // the thread whose partner this node is
#pragma unroll
            for (int c = 0; c < 5; ++c) acc[tw][0][c] = fx_add(acc[tw][0][c], fx_sub(G[c], get(G[c], from)));
          }
        } else {
          {  // the own pair
            Node B;
            load(so[tw][1], B);
            fx64 G[5];
            pair(0, B, sb.Q[pos + TPL + n * pos], G);
#pragma unroll
            for (int c = 0; c < 5; ++c) {
              const fx64 x = c == 0 ? G[c] : fx_unbias64(G[c], c == 4 ? sh.hE : sh.hG[c - 1]);
              acc[tw][0][c] = fx_add(acc[tw][0][c], x);
              acc[tw][1][c] = fx_sub(acc[tw][1][c], x);
            }
          }
#pragma unroll
          for (int s = 1; s <= (TPL - 1) / 2; ++s) {
            const int b = pos + s < TPL ? pos + s : pos + s - TPL;
            const int from = lane + (pos >= s ? -s : TPL - s);
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              const int bx = b + x * TPL;
              Node B;
              load(vsw<NP>(base + bx * step), B);
              fx64 G0[5], G1[5];
              pair(0, B, sb.Q[bx + n * pos], G0);
              pair(1, B, sb.Q[bx + n * (pos + TPL)], G1);
#pragma unroll
              for (int c = 0; c < 5; ++c) {
                acc[tw][0][c] = fx_add(acc[tw][0][c], G0[c]);
                acc[tw][1][c] = fx_add(acc[tw][1][c], G1[c]);
                acc[tw][x][c] = fx_sub(acc[tw][x][c], get(fx_add(G0[c], G1[c]), from));
              }
            }
          }
          if constexpr (TPL % 2 == 0) {
            // the thread n/4 places on: this thread's first node with its first, second with second; the
            // threads of the line's second half take the other two pairs (first with second)
            constexpr int s = TPL / 2;
            const bool up = pos >= s;
            const int b = up ? pos - s : pos + s, from = lane + (up ? -s : s);
            const int b0 = up ? b + TPL : b, b1 = up ? b : b + TPL;
            fx64 G0[5], G1[5];
            {
              Node B;
              load(vsw<NP>(base + b0 * step), B);
              pair(0, B, sb.Q[b0 + n * pos], G0);
            }
            {
              Node B;
              load(vsw<NP>(base + b1 * step), B);
              pair(1, B, sb.Q[b1 + n * (pos + TPL)], G1);
            }
#pragma unroll
            for (int c = 0; c < 5; ++c) {
              // what the other thread's pairs give this thread's first and second node
              const fx64 r0 = get(up ? G1[c] : G0[c], from), r1 = get(up ? G0[c] : G1[c], from);
              acc[tw][0][c] = fx_add(acc[tw][0][c], fx_sub(G0[c], r0));
              acc[tw][1][c] = fx_add(acc[tw][1][c], fx_sub(G1[c], r1));
            }
          }
        }
      }
      __syncthreads();  // the direction's metric terms and viscous fluxes are read
#pragma unroll
      for (int tw = 0; tw < C::TPW; ++tw) {
        const int li = (warp + tw * C::NW) * C::LPW + lsub;
        if (lsub < C::LPW && li < n2) {
#pragma unroll
          for (int o = 0; o < OWN; ++o)
#pragma unroll
            for (int c = 0; c < 5; ++c) Ad[c * n3 + so[tw][o]] = acc[tw][o][c];
        }
      }
    }
    __syncthreads();

    // ---- face fluxes onto the end nodes of their lines (a direction's two faces share no node)
    for (int t = tid; t < 6 * n2; t += NT) {
      const int ls = t / n2 + 1, ab = t - (ls - 1) * n2;
      const int a = ab % n, b = ab / n;
      const int side = es[2 * (ls - 1)], flip = es[2 * (ls - 1) + 1];
      int p, q;
      s2v2_inv(N, a, b, flip, ls, p, q);
      const double* f = Flux + (size_t)side * 5 * n2 + p + n * q;
      const int dir = ls == L_XI_MINUS || ls == L_XI_PLUS ? 0 : (ls == L_ETA_MINUS || ls == L_ETA_PLUS ? 1 : 2);
      fx64* const o = A + (6 + dir * DS) * n3 + vsw<NP>(face_node(n, ls, a, b, is_minus(ls) ? 0 : N));
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        const fx64 x = fx_from(f[v * n2], fx_r0(sc.d[dir].t[v] + (v == 0 ? 2 : 3)));
        o[v * n3] += flip == 0 ? x : -x;
      }
    }
    __syncthreads();

    // ---- 1/w of the three directions, -1, the Jacobian
#pragma unroll
    for (int it = 0; it < NPT; ++it) {
      const int node = tid + it * NT;
      if (node < n3) {
        const int i = node % n, j = (node / n) % n, k = node / n2;
        const FxLimb w[3] = {sb.iw[i], sb.iw[j], sb.iw[k]};
        const fx64* const a = A + vsw<NP>(node);
        const double c = -iw0 * Me[9 * n3 + node];
        const int ch = __double2hiint(c), cl = __double2loint(c);
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          fx64 m = 0;
          FxLimb x[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            // to the smallest of the three directions' scales, halved for the range of the sum
            x[d] = fx_limb(fx_sar(a[(6 + d * DS + v) * n3], min(sc.d[d].t[v] - sc.t[v] + 1, 63)));
            m = fx_mid(x[d], w[d], m);
          }
          fx64 t = m >> 32;
#pragma unroll
          for (int d = 0; d < 3; ++d) t = fx_mad(x[d].h, w[d].h, t);
          Us[node * 5 + v] = fx_to_double(t, m) * __hiloint2double(ch - ((sc.t[v] + (v == 0 ? 2 : 3) - 5) << 20), cl);
        }
      }
    }
  } else {
    vol_block_fp64<NP, SPLIT, PARAB, NT>(Ue, Pe, Ge, Me, Flux, es, basis, 0, gas.mu, gas.lambda,
                                         reinterpret_cast<double*>(sb.Q), Us);
  }
  __syncthreads();
  // output / LSERK-W2 stage, one value per thread in turn (the element's record is contiguous)
  const size_t g0 = (size_t)e * 5 * n3;
  for (int t = tid; t < 5 * n3; t += NT) {
    const double val = Us[t];
    if (rkmode == 0) {
      rk.Ut[g0 + t] = val;
    } else {
      const double utmp = rk.Ut_tmp[g0 + t] * rk.mRKA + val;
      rk.Ut_tmp[g0 + t] = utmp;
      rk.U[g0 + t] = rk.U[g0 + t] + utmp * rk.b_dt;
    }
  }
}

}  // namespace gx

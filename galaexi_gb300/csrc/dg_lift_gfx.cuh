// k_lift_gfx: the lifting of the FP64 form on Gauss nodes (BR1, BR2) and BR2 on Gauss-Lobatto nodes, strong
// non-conservative form, in block fixed-point arithmetic on the integer pipes (dg_fx.cuh).
//
// Lifting_VolInt_Nonconservative (src/dg/lifting_volint.t90:262-328), the surface part
// (lifting_fillflux.t90:39-103, 212-256, surfint.t90:591-725), ProlongToFaceLifting and the BR2 traces
// (Lifting_SurfInt_BR2, lifting_br2.t90:191-310) of u, v, w, T.  k_lift spends about 360 FP64 instructions per
// node on this at N = 5 (65 cycles each per warp and sub-partition); here the derivatives, the face fluxes
// F = 0.5 SurfElem n (P_slave - P_master), the node sums g = sJ (sum_dir M_dir y_dir + Lhat- F- + Lhat+ F+) and
// the traces are integer multiply-adds, and the FP64 pipe only converts the results.
//
// Mapping: one element per block, three passes over shared memory: one thread per line and variable
// differentiates (even and odd parts, as in k_lift_fx) while the face nodes' threads have left the fluxes;
// one thread per node adds up; one thread per line and variable prolongs to the line's two faces, again with
// even and odd parts, which gives both traces for the products of one.  Bound by the integer pipes (issue 53%,
// ALU 56% at N = 5 and 7; the conversions to integers on the FP64 pipe instead made it 4% slower).  k_lift and
// now: N = 5, 24^3 curved, Gauss BR2 2.04 -> 0.629 ms; Gauss BR1 N = 2, 64^3 4.69 -> 2.43, N = 4, 32^3
// 2.15 -> 0.851, N = 7, 20^3 2.20 -> 0.729, N = 9, 16^3 3.17 -> 0.919; Gauss-Lobatto BR2 N = 7, 24^3 2.75 -> 1.22.
#pragma once
#include "dg_fx.cuh"
#include "dg_kernels.cuh"
#include "dg_lift_fx.cuh"

namespace gx {

template <int NP> struct LiftGfx {
  // threads: whole passes over the 12 n^2 lines and the n^3 nodes, and enough warps beside the shared memory (one
  // thread for each of the 12 n^2 lines of small elements: N = 2 3.33 ms, N = 3, 48^3 2.59 against 1.48)
  static constexpr int NT = NP <= 4 ? 64 : (NP == 5 ? 160 : (NP == 6 ? 224 : (NP == 7 ? 352 : (NP == 8 ? 256 : 512))));
  static constexpr size_t smem = sizeof(fx64) * (17 * NP * NP * NP + 78 * NP * NP) + sizeof(int) * 6 * NP * NP;
  static constexpr int byreg = NT == 512 ? 1 : 704 / NT, bysm = (int)((227 * 1024) / (smem + 2048));
  static constexpr int MINB = bysm < 1 ? 1 : (byreg < bysm ? byreg : bysm);
};
// D as in LiftFxBasis; Lh: L_hat of the plus face (minus: mirrored) times 2^sL; te, to: L of the plus face in
// even and odd parts (odd n: te's last is the middle node's) times 2^sT; LL: eta_BR2 L L_hat (plus) times 2^sLL
template <int NP> struct LiftGfxBasis {
  static constexpr int H = NP / 2, HE = (NP + 1) / 2;
  LiftFxBasis<NP> d;
  FxDig Lh[NP], te[HE], to[H], LL[NP];
  int sL, sT, sLL;
};

// one variable: shifts of y and F to the range, exponent of its gradients; scale of its traces, shifts of their two
// parts
struct LiftGfxScale {
  int KY, KF, kG, s_o, kt, kb;
};

// The FP64 lifting by the block (elements whose values do not fit one scale; FP64-issue bound like k_lift: all elements
// of 20^3, N = 5, Gauss BR1 and BR2 0.91 and 1.16 ms, k_lift 1.01 and 1.19): the gradients to Gvol, those that the
// traces are formed from (BR2: the volume part) to Y.  X, F: shared memory as in the kernel below
template <int NP, bool GAUSS, bool BR2, int NT>
__device__ __noinline__ void lift_gen_fp64(const double* Pe, const double* Me, const double* Pf, const double* Fgeo,
                                           const int* es, int nSides, const double* D, const double* Lhm,
                                           const double* Lhp, double* Ge, double* X, double* F, double* Y) {
  constexpr int n = NP, n2 = NP * NP, n3 = NP * NP * NP, N = NP - 1;
  const int liftc[4] = {1, 2, 3, 5};
#pragma unroll 1
  for (int t = threadIdx.x; t < 6 * n2; t += NT) {
    const int f = t / n2, ab = t - f * n2, dir = f >> 1, pm = f & 1;
    const int ls = dir == 0 ? (pm == 0 ? L_XI_MINUS : L_XI_PLUS)
                            : (dir == 1 ? (pm == 0 ? L_ETA_MINUS : L_ETA_PLUS) : (pm == 0 ? L_ZETA_MINUS : L_ZETA_PLUS));
    const int side = es[2 * (ls - 1)], flip = es[2 * (ls - 1) + 1];
    int p, q;
    s2v2_inv(N, ab % n, ab / n, flip, ls, p, q);
    const double* const pl = Pf + (size_t)side * 6 * n2 + p + n * q;
    const double* const pr = pl + (size_t)nSides * 6 * n2;
    const double* const fg = Fgeo + (size_t)side * 10 * n2 + p + n * q;
    const double w = 0.5 * fg[9 * n2], nv[3] = {w * fg[0], w * fg[n2], w * fg[2 * n2]};
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const double fl = pr[liftc[v] * n2] - pl[liftc[v] * n2];
#pragma unroll
      for (int d = 0; d < 3; ++d) F[(f * 12 + d * 4 + v) * n2 + ab] = fl * nv[d];
    }
  }
  lift_lines_fp64<NP, NT>(Pe, D, X, Y);
#pragma unroll 1
  for (int node = threadIdx.x; node < n3; node += NT) {
    double g[12];
    lift_node_fp64<NP>(Me, Y, node, g);
    if constexpr (BR2)
#pragma unroll
      for (int c = 0; c < 12; ++c) Y[c * n3 + vsw<NP>(node)] = g[c];
    const double sj = Me[(size_t)9 * n3 + node];
    const int ijk[3] = {node % n, (node / n) % n, node / n2};
    const int ab[3] = {ijk[1] + n * ijk[2], ijk[0] + n * ijk[2], ijk[0] + n * ijk[1]};
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const int dir = f >> 1, l = ijk[dir];
      if (!GAUSS && l != ((f & 1) == 0 ? 0 : N)) continue;
      const double w = sj * ((f & 1) == 0 ? Lhm[l] : Lhp[l]);
#pragma unroll
      for (int c = 0; c < 12; ++c) g[c] = g[c] + w * F[(f * 12 + c) * n2 + ab[dir]];
    }
#pragma unroll
    for (int c = 0; c < 12; ++c) {
      Ge[(c / 4 * 5 + 1 + c % 4) * n3 + node] = g[c];
      if constexpr (!BR2) Y[c * n3 + vsw<NP>(node)] = g[c];
    }
  }
}

template <int NP, bool GAUSS, bool BR2>
__global__ void __launch_bounds__(LiftGfx<NP>::NT, LiftGfx<NP>::MINB)
k_lift_gfx(const double* __restrict__ Pvol, const double* __restrict__ Met, const float* __restrict__ MetL,
           const double* __restrict__ Pf, const double* __restrict__ Fgeo, const int* __restrict__ E2S,
           const __grid_constant__ LiftGfxBasis<NP> gb, DevBasis<double> basis, double eta, int nSides,
           double* __restrict__ Gvol, double* __restrict__ Gf) {
  using C = LiftGfx<NP>;
  constexpr int n = NP, n2 = NP * NP, n3 = NP * NP * NP, N = NP - 1, NT = C::NT;
  constexpr int H = LiftGfxBasis<NP>::H, HE = LiftGfxBasis<NP>::HE;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  fx64* const Y = reinterpret_cast<fx64*>(smem_raw);       // [3][4][n3]: derivatives, then gradients
  fx64* const X = Y + 12 * n3;                             // [4][n3]: u, v, w, T
  fx64* const F = X + 4 * n3;                              // [3][2][12][n2]: face fluxes
  fx64* const Cb = F + 72 * n2;                            // [3][2][n2]: eta sum_l L Lhat sJ (BR2)
  fx64* const J = Cb + 6 * n2;                             // [n3]: sJ
  int* const off = reinterpret_cast<int*>(J + n3);         // [3][2][n2]: the face nodes' places on their sides
  __shared__ unsigned mag[4], magY[4], magF[4];
  __shared__ LiftGfxScale sc[4];
  __shared__ int es[12], cold;
  __shared__ FxDig Lh[NP];
  const int e = blockIdx.x, tid = threadIdx.x;
  if (tid < 4) mag[tid] = magY[tid] = magF[tid] = 0u;
  if (tid == 4) cold = 0;
  if (tid < 12) es[tid] = E2S[(size_t)e * 12 + tid];
  if (tid >= 32 && tid < 32 + n) Lh[tid - 32] = gb.Lh[tid - 32];
  __syncthreads();
  const double* const Pe = Pvol + (size_t)e * 7 * n3;
  const double* const Me = Met + (size_t)e * 10 * n3;
  const float* const ml = MetL + (size_t)e * kMetL;
  auto liftc = [](int v) { return v == 3 ? 5 : v + 1; };
  auto side_of = [](int dir, int pm) {
    return dir == 0 ? (pm == 0 ? L_XI_MINUS : L_XI_PLUS)
                    : (dir == 1 ? (pm == 0 ? L_ETA_MINUS : L_ETA_PLUS) : (pm == 0 ? L_ZETA_MINUS : L_ZETA_PLUS));
  };
  // node l of line (a, b) of a direction
  auto line = [](int dir, int ab) { return dir == 0 ? n * ab : (dir == 1 ? (ab % n) + n2 * (ab / n) : ab); };
  bool ok = ml[0] < 200.f && ml[12] < 200.f;
  int sM[3];  // of M_dir,d and SurfElem n_d, for each component d of the gradient
#pragma unroll
  for (int d = 0; d < 3; ++d) sM[d] = ok ? 58 - ((int)floorf(ml[14 + d]) + 1) : 0;
  const int sJ = ok ? 59 - ((int)floorf(ml[13]) + 1) : 0;
  // ---- one scale per variable: the largest magnitude of the element and of both traces on its faces
  {
    unsigned m[4] = {0u, 0u, 0u, 0u};
#pragma unroll 2
    for (int node = tid; node < n3; node += NT) {
      J[node] = fd_pack(fd_from(Me[9 * n3 + node], fx_r0(sJ)));
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const double x = Pe[liftc(v) * n3 + node];
        X[v * n3 + vsw<NP>(node)] = __double_as_longlong(x);
        m[v] = max(m[v], fx_mag(x));
      }
    }
#pragma unroll 2
    for (int t = tid; t < 6 * n2; t += NT) {
      const int f = t / n2;
      const double* const pl = Pf + (size_t)es[2 * f] * 6 * n2 + t - f * n2;
      const double* const pr = pl + (size_t)nSides * 6 * n2;
#pragma unroll
      for (int v = 0; v < 4; ++v) m[v] = max(m[v], max(fx_mag(pl[liftc(v) * n2]), fx_mag(pr[liftc(v) * n2])));
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) fx_block_max(m[v], &mag[v]);
  }
  __syncthreads();
  ok = ok && lift_fits(mag);
  // Scales (powers of two): |x| < 2^57, |M| < 2^58 and SurfElem n < 2^58 for each component of the gradient (in flat
  // elements they differ by the aspect ratio), |sJ| < 2^59; y = D x below 2^60 (as in
  // k_lift_fx), F = (SurfElem/2 n) dx below 2^59.  From here on the scale follows the largest |y| and |F| of the
  // element, which are smaller than their bounds by the smoothness of the field (with the bounds alone 4 to 16
  // times the FP64 kernel's error on smooth viscous flow): y and F are shifted to one scale of the sums M y (three
  // terms) and Lhat F (six), |y| < 2^60 and |F| < 2^59, so that the sums stay below 2^60.6 and, times sJ, 2^59.6;
  // sums and differences of two in the traces then fit digits.
  if (ok) {
    int r0[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) r0[v] = fx_r0(57 - fx_exp(mag[v]));
#pragma unroll 1
    for (int node = tid; node < n3; node += NT)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        fx64* const x = X + v * n3 + vsw<NP>(node);
        const double d = __longlong_as_double(*x);
        if (v == 3 && lift_cold(d, mag[3])) cold = 1;
        *x = fd_pack(fd_from(d, r0[v]));
      }
    // ---- face fluxes, and the BR2 weights of the lines
    unsigned mf[4] = {0u, 0u, 0u, 0u}, my[4] = {0u, 0u, 0u, 0u};
#pragma unroll 1
    for (int t = tid; t < 6 * n2; t += NT) {
      const int f = t / n2, ab = t - f * n2, a = ab % n, b = ab / n, dir = f >> 1, ls = side_of(dir, f & 1);
      const int side = es[2 * (ls - 1)], flip = es[2 * (ls - 1) + 1];
      int p, q;
      s2v2_inv(N, a, b, flip, ls, p, q);
      off[t] = p + n * q;
      const double* const pl = Pf + (size_t)side * 6 * n2 + p + n * q;
      const double* const pr = pl + (size_t)nSides * 6 * n2;
      const double* const fg = Fgeo + (size_t)side * 10 * n2 + p + n * q;
      FxDig dx[4], G[3];
#pragma unroll
      for (int v = 0; v < 4; ++v) dx[v] = fd_from(pr[liftc(v) * n2], r0[v]) - fd_from(pl[liftc(v) * n2], r0[v]);
      const int es9 = fx_exp(fx_mag(fg[9 * n2]));
      const FxDig se = fd_from(fg[9 * n2], fx_r0(58 - es9));
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        // SurfElem and n_d with all their bits, then to the component's scale
        const double nd = fg[d * n2];
        const int en = fx_exp(fx_mag(nd));
        FxDot s;
        s.add(fd_from(nd, fx_r0(58 - en)), se);
        G[d] = fd_scaled(s.sum<2>(), max(sM[d] - (58 - es9 - en), -63));
      }
      fx64* const Fo = F + f * 12 * n2 + ab;
#pragma unroll
      for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          FxDot s;
          s.add(dx[v], G[d]);
          const fx64 x = s.sum<3>();
          mf[v] = max(mf[v], fx_mag64(x));
          Fo[(d * 4 + v) * n2] = x;
        }
      if constexpr (BR2) {
        const int base = line(dir, ab), step = dir == 0 ? 1 : (dir == 1 ? n : n2);
        FxDot s;
        if constexpr (GAUSS) {
#pragma unroll
          for (int l = 0; l < n; ++l) {
            if (l == 4 || l == 8) s.carry();
            s.add(fd_unpack(J[base + ((f & 1) ? l : N - l) * step]), gb.LL[l]);
          }
        } else {
          s.add(fd_unpack(J[base + ((f & 1) ? N : 0) * step]), gb.LL[N]);
        }
        Cb[f * n2 + ab] = fd_pack(fd_split(s.sum()));
      }
    }
    __syncthreads();
    // ---- derivatives
#pragma unroll 1
    for (int task = tid; task < 12 * n2; task += NT) {
      const int dv = task / n2, li = task - dv * n2, dir = dv >> 2, v = dv & 3;
      const int step = dir == 0 ? 1 : (dir == 1 ? n : n2), base = line(dir, li);
      const fx64* const Xv = X + v * n3;
      auto at = [&](int l) {
        return fd_unpack(Xv[vsw<NP>(base + l * step)]);
      };
      FxDig ev[HE], od[H];
#pragma unroll
      for (int l = 0; l < H; ++l) {
        const FxDig a = at(l), b = at(N - l);
        ev[l] = a + b;
        od[l] = a - b;
      }
      if constexpr (NP % 2) ev[H] = at(H);
      fx64* const Yo = Y + dv * n3;
      unsigned m = 0u;
#pragma unroll
      for (int i = 0; i < H; ++i) {
        FxDot A, B;
#pragma unroll
        for (int l = 0; l < HE; ++l) {
          if (l == 4) A.carry();
          A.add(ev[l], gb.d.even[i][l]);
        }
#pragma unroll
        for (int l = 0; l < H; ++l) {
          if (l == 4) B.carry();
          B.add(od[l], gb.d.odd[i][l]);
        }
        const fx64 a = A.sum<3>(), b = B.sum<3>(), y0 = a + b, yN = b - a;
        m = max(m, max(fx_mag64(y0), fx_mag64(yN)));
        Yo[vsw<NP>(base + i * step)] = y0;
        Yo[vsw<NP>(base + (N - i) * step)] = yN;
      }
      if constexpr (NP % 2) {
        FxDot B;
#pragma unroll
        for (int l = 0; l < H; ++l) B.add(od[l], gb.d.odd[H][l]);
        const fx64 y = B.sum<3>();
        m = max(m, fx_mag64(y));
        Yo[vsw<NP>(base + H * step)] = y;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) my[c] = max(my[c], v == c ? m : 0u);
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      fx_block_max(my[v], &magY[v]);
      fx_block_max(mf[v], &magF[v]);
    }
    __syncthreads();
    {
      const int v = tid & 3, ev = fx_exp(mag[v]), bY = fx_bits(magY[v]), bF = fx_bits(magF[v]);
      // (without the components' sM)
      const int s_v = gb.d.sD - ev - 60, s_F = 1 - ev, s_s = s_F + gb.sL - 60;  // of M y / 2^60, Lhat F / 2^60
      const int s_g = min(s_v + min(60 - bY, 30), s_s + min(59 - bF, 30)), s_G = s_g + sJ - 60;
      LiftGfxScale o;
      o.KY = max(s_g - s_v, -63);
      o.KF = max(s_g - s_s, -63);
      o.kG = -s_G;
      // traces (two bits more than the product with L): below 2^61; F times the BR2 weight (< 2^58) below 2^57
      const int s_t = s_G + (GAUSS ? gb.sT - 58 : 0), s_b = s_F + o.KF + gb.sLL + sJ - 120;
      o.s_o = BR2 ? min(s_t, s_b) : s_t;
      o.kt = min(s_t - o.s_o, 63);
      o.kb = min(s_b - o.s_o, 63);
      if (tid < 4) sc[tid] = o;
      int KF[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) KF[c] = __shfl_sync(0xffffffffu, o.KF, c);
#pragma unroll 1
      for (int t = tid; t < 6 * n2; t += NT) {
        const int f = t / n2;
        fx64* const Fo = F + f * 11 * n2 + t;  // f 12 n2 + ab
#pragma unroll
        for (int c = 0; c < 12; ++c) Fo[c * n2] = fd_pack(fd_scaled(Fo[c * n2], KF[c & 3]));
      }
    }
    __syncthreads();
    ok = cold == 0;
    // ---- node by node
#pragma unroll 1
    for (int node = ok ? tid : n3; node < n3; node += NT) {
      const int i = node % n, j = (node / n) % n, k = node / n2, sn = vsw<NP>(node);
      const int ix[3] = {i, j, k}, ab[3] = {j + n * k, i + n * k, i + n * j};
      FxDig M[9];
#pragma unroll
      for (int c = 0; c < 9; ++c) M[c] = fd_from(Me[c * n3 + node], fx_r0(sM[c % 3]));
      const FxDig jc = fd_unpack(J[node]);
      FxDig lm[3], lp[3];
      if constexpr (GAUSS) {
#pragma unroll
        for (int dir = 0; dir < 3; ++dir) { lm[dir] = Lh[N - ix[dir]]; lp[dir] = Lh[ix[dir]]; }
      }
      const FxDig le = Lh[N];
      double* const G = Gvol + (size_t)e * 15 * n3 + node;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const LiftGfxScale o = sc[v];
        FxDig y[3];
#pragma unroll
        for (int dir = 0; dir < 3; ++dir) y[dir] = fd_scaled(Y[(dir * 4 + v) * n3 + sn], o.KY);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          FxDotU p;
#pragma unroll
          for (int dir = 0; dir < 3; ++dir) p.add(y[dir], M[3 * dir + d]);
          const fx64 vol = p.sum();
#pragma unroll
          for (int dir = 0; dir < 3; ++dir) {
            const fx64* const Fd = F + (dir * 24 + d * 4 + v) * n2 + ab[dir];
            if constexpr (GAUSS) {
              p.add(fd_unpack(Fd[0]), lm[dir]);
              p.add(fd_unpack(Fd[12 * n2]), lp[dir]);
            } else if (ix[dir] == 0 || ix[dir] == N) {
              p.add(fd_unpack(Fd[ix[dir] == 0 ? 0 : 12 * n2]), le);
            }
          }
          FxDotU g;
          g.add(fd_split(p.sum()), jc);
          const fx64 gt = g.sum();
          G[(d * 5 + 1 + v) * n3] = fx_scaled(gt, o.kG - sM[d]);
          // for the traces: BR2 prolongs the volume part only
          if constexpr (BR2) {
            FxDotU h;
            h.add(fd_split(vol), jc);
            Y[(d * 4 + v) * n3 + sn] = h.sum();
          } else {
            Y[(d * 4 + v) * n3 + sn] = gt;
          }
        }
      }
    }
  }
  if (!ok) {
    lift_gen_fp64<NP, GAUSS, BR2, NT>(Pe, Me, Pf, Fgeo, es, nSides, basis.D, basis.Lhm, basis.Lhp,
                                      Gvol + (size_t)e * 15 * n3, reinterpret_cast<double*>(X),
                                      reinterpret_cast<double*>(F), reinterpret_cast<double*>(Y));
  }
  __syncthreads();
  // ---- traces on the two faces of a line
#pragma unroll 1
  for (int task = tid; task < 12 * n2; task += NT) {
    const int dv = task / n2, li = task - dv * n2, dir = dv >> 2, v = dv & 3;
    const int step = dir == 0 ? 1 : (dir == 1 ? n : n2), base = line(dir, li);
    int at[2], sd[2];
    double* out[2];
#pragma unroll
    for (int pm = 0; pm < 2; ++pm) {
      const int ls = side_of(dir, pm), side = es[2 * (ls - 1)], flip = es[2 * (ls - 1) + 1];
      if (ok) {
        at[pm] = off[(dir * 2 + pm) * n2 + li];
      } else {
        int p, q;
        s2v2_inv(N, li % n, li / n, flip, ls, p, q);
        at[pm] = p + n * q;
      }
      sd[pm] = side;
      out[pm] = Gf + ((size_t)(flip == 0 ? 0 : 1) * nSides + side) * 15 * n2 + (1 + v) * n2 + at[pm];
    }
    if (ok) {
      const LiftGfxScale o = sc[v];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const fx64* const g = Y + (d * 4 + v) * n3;
        fx64 tr[2];
        if constexpr (GAUSS) {
          FxDot E, O;
#pragma unroll
          for (int l = 0; l < H; ++l) {
            const fx64 a = g[vsw<NP>(base + l * step)], b = g[vsw<NP>(base + (N - l) * step)];
            if (l == 4) { E.carry(); O.carry(); }
            E.add(fd_split(a + b), gb.te[l]);
            O.add(fd_split(a - b), gb.to[l]);
          }
          if constexpr (NP % 2) E.add(fd_split(g[vsw<NP>(base + H * step)]), gb.te[H]);
          const fx64 ee = E.sum<2>(), oo = O.sum<2>();
          tr[0] = ee - oo;
          tr[1] = ee + oo;
        } else {
          tr[0] = g[vsw<NP>(base)];
          tr[1] = g[vsw<NP>(base + N * step)];
        }
#pragma unroll
        for (int pm = 0; pm < 2; ++pm) {
          fx64 t = tr[pm];
          if constexpr (BR2) {
            FxDotU s;
            s.add(fd_unpack(F[((dir * 2 + pm) * 12 + d * 4 + v) * n2 + li]), fd_unpack(Cb[(dir * 2 + pm) * n2 + li]));
            t = fx_sar(t, o.kt) + fx_sar(s.sum(), o.kb);
          }
          out[pm][d * 5 * n2] = fx_scaled(t, -o.s_o - sM[d]);
        }
      }
    } else {
#pragma unroll 1
      for (int pm = 0; pm < 2; ++pm) {
        const double* const Lv = pm == 0 ? basis.Lm : basis.Lp;
        const double* const Lw = pm == 0 ? basis.Lhm : basis.Lhp;
        const int l0 = GAUSS ? 0 : (pm == 0 ? 0 : N), l1 = GAUSS ? N : l0;
        const double* const fg = Fgeo + (size_t)sd[pm] * 10 * n2 + at[pm];
        double bw = 0.;
        if constexpr (BR2) {
          const double* const pl = Pf + ((size_t)sd[pm] * 6 + liftc(v)) * n2 + at[pm];
          for (int l = l0; l <= l1; ++l) bw = bw + Lv[l] * Lw[l] * Me[9 * n3 + base + l * step];
          bw = eta * 0.5 * fg[9 * n2] * bw * (pl[(size_t)nSides * 6 * n2] - pl[0]);
        }
#pragma unroll 1
        for (int d = 0; d < 3; ++d) {
          double s = 0.;
          for (int l = l0; l <= l1; ++l) s = s + __longlong_as_double(Y[(d * 4 + v) * n3 + vsw<NP>(base + l * step)]) * (GAUSS ? Lv[l] : 1.);
          if constexpr (BR2) s = s + bw * fg[d * n2];
          out[pm][d * 5 * n2] = s;
        }
      }
    }
  }
}

}  // namespace gx

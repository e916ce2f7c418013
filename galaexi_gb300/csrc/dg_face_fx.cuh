// k_face_dp: FillFlux (src/dg/fillflux.f90:45-172) of the connected sides in the FP64 form: Riemann flux
// (riemann.f90:216-289, 707-1257), BR1 viscous flux (riemann.f90:594-700, flux.f90:779-847) and SurfElem, one
// thread per face node, for the solvers LF, Roe, Roe with entropy fix and HLLC and the central parts of the
// weak form, PI and KG; the others run in k_face.
//
// Bound by the FP64 issue rate (65 cycles per warp instruction and sub-partition), so it is written for few
// FP64 instructions:
//   * no rotation into the face frame: the solvers only need the normal velocity, the tangential parts of
//     the jumps are v - (v.n) n, so the tangents are neither read nor applied;
//   * sound speeds of the states from the stored temperature, c^2 = kappa R T (the enthalpies (E + p) (1/rho) as
//     the volume kernel forms them: cp T + |v|^2/2 is shorter, but its rounding does not cancel against the
//     volume's, which cost up to three times the error);
//   * Roe averages from one square root and one reciprocal: rho~ = sqrt(rho_L rho_R), weight of the right
//     state rho_R / (rho_R + rho~); c and 1/c^2 from one reciprocal square root;
//   * reciprocals and square roots by Newton's iteration (two steps) from the FP32 approximation, with the
//     exponents handled by integer instructions; comparisons on the bit patterns;
//   * Roe's wave strengths from the jumps of the conserved variables, in vector form;
//   * the viscous traction tau n from the symmetrised gradient, its momentum part added up over both sides.
#pragma once
#include "dg_dp.cuh"
#include "dg_kernels.cuh"

namespace gx {

struct FaceGas {
  double kappaM1, kR, mu, lambda;  // kR = kappa R
};
struct FaceSide {
  double rho, v[3], p, T, un, E, srho;
};

// central part: CENTRAL -1: mean of the Euler fluxes (EvalEulerFlux1D_fast, flux.f90:1123-1143), else the split
// surface flux (splitflux.f90:270-761)
template <int CENTRAL>
__device__ __forceinline__ void central_flux(const FaceSide& L, const FaceSide& R, const double n[3], double HL,
                                             double HR, double F[5]) {
  const double ps = 0.5 * (L.p + R.p);
  if constexpr (CENTRAL < 0) {
    const double mL = 0.5 * L.rho * L.un, mR = 0.5 * R.rho * R.un;
    F[0] = mL + mR;
#pragma unroll
    for (int c = 0; c < 3; ++c) F[1 + c] = mL * L.v[c] + (mR * R.v[c] + ps * n[c]);
    F[4] = mL * HL + mR * HR;
  } else {
    const double us = L.un + R.un, q = 0.125 * (L.rho + R.rho) * us;
    F[0] = 2. * q;
#pragma unroll
    for (int c = 0; c < 3; ++c) F[1 + c] = q * (L.v[c] + R.v[c]) + ps * n[c];
    if constexpr (CENTRAL == DG_SPLIT_PI) F[4] = q * (HL + HR);
    else F[4] = q * (L.E * L.srho + R.E * R.srho) + 0.5 * ps * us;
  }
}

template <int RIEM, int CENTRAL>
__device__ __forceinline__ void riemann_dp(const double dm[3], const FaceSide& L, const FaceSide& R,
                                           const double n[3], const FaceGas& g, double F[5]) {
  const double HL = (L.E + L.p) * L.srho, HR = (R.E + R.p) * R.srho;
  if constexpr (RIEM == DG_RIEMANN_LF) {
    central_flux<CENTRAL>(L, R, n, HL, HR, F);
    // |u_n| + c: the larger temperature has the larger sound speed
    const double c2 = g.kR * dp_max(L.T, R.T);
    const double hl = 0.5 * (dp_max(dp_abs(L.un), dp_abs(R.un)) + dp_sqrt(c2));
    F[0] = F[0] - hl * (R.rho - L.rho);
#pragma unroll
    for (int c = 0; c < 3; ++c) F[1 + c] = F[1 + c] - hl * dm[c];
    F[4] = F[4] - hl * (R.E - L.E);
    return;
  }
  // Roe averages
  double rr = L.rho * R.rho;
  // (two negative densities: no square root)
  rr = __hiloint2double(__double2hiint(rr) | (__double2hiint(L.rho) & (int)0x80000000), __double2loint(rr));
  // (a product outside the helpers' range: the roots one by one, densities of 1e-150 or 1e150 would leave FP64's)
  const double rt = dp_exponent_in(rr, 123, 1800) ? dp_sqrt(rr) : dp_sqrt_rare(L.rho) * dp_sqrt_rare(R.rho);
  const double w = R.rho * dp_rcp(R.rho + rt);
  const double un = fma(w, R.un - L.un, L.un);
  double u[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) u[c] = fma(w, R.v[c] - L.v[c], L.v[c]);
  const double H = fma(w, HR - HL, HL);
  const double q2 = 0.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
  const double c2 = g.kappaM1 * (H - q2);
  double ic;
  const double c = dp_root<false>(c2, ic);
  if constexpr (RIEM == DG_RIEMANN_HLLC) {
    const double Sl = un - c, Sr = un + c;
    const double mnL = L.rho * (Sl - L.un), mnR = R.rho * (Sr - R.un);
    const double Ss = dp_div((R.p - L.p) + mnL * L.un - mnR * R.un, mnL - mnR);
    const bool superL = dp_ge0(Sl), superR = dp_le0(Sr);
    const bool left = superL || (!superR && dp_ge0(Ss));
    const double rho = left ? L.rho : R.rho, p = left ? L.p : R.p, us = left ? L.un : R.un;
    const double E = left ? L.E : R.E, S = left ? Sl : Sr;
    // with k = (Ss - u) / (S - Ss) the star state's jumps are U* - U = k U + ..., without the difference of two states:
    //   rho* = rho (1 + k),  S (E* - E) = S k (E + p) + S rho* (Ss - u) Ss
    const bool super = superL || superR;
    const double dus = Ss - us, k = dus * dp_rcp(S - Ss);
    const double ust = super ? us : fma(S, k, us), b = super ? 0. : S * (fma(rho, k, rho) * dus);
    F[0] = rho * ust;
    const double pn = p + b;
#pragma unroll
    for (int c = 0; c < 3; ++c) F[1 + c] = (left ? L.v[c] : R.v[c]) * F[0] + pn * n[c];
    F[4] = (E + p) * ust + (super ? 0. : b * Ss);
    return;
  }
  central_flux<CENTRAL>(L, R, n, HL, HR, F);
  double l1 = un - c, l2 = un, l5 = un + c;
  if constexpr (RIEM == DG_RIEMANN_ROEENTROPYFIX) {
    const double aL = g.kR * L.T, aR = g.kR * R.T;
    const double cL = dp_sqrt(aL), cR = dp_sqrt(aR);
    auto fix = [](double a, double al, double ar) {
      const double da = dp_max(dp_max(a - al, ar - a), 0.), ab = dp_abs(a);
      return dp_bits(ab) < dp_bits(da) ? 0.5 * (dp_div(a * a, da) + da) : ab;
    };
    l1 = fix(l1, L.un - cL, R.un - cR);
    l2 = fix(l2, L.un, R.un);
    l5 = fix(l5, L.un + cL, R.un + cR);
  } else {
    l1 = dp_abs(l1); l2 = dp_abs(l2); l5 = dp_abs(l5);
  }
  // half the wave strengths times the eigenvalues, from the jumps of the conserved variables (the pressure's
  // own round-off would enter the strengths with a jump of p): with dr, dm, dE
  //   dp = (kappa-1) (dE - u.dm + |u|^2/2 dr),  ds = dm - u dr,  dsn = ds.n  (rho~ dv and rho~ dv.n)
  const double dr = R.rho - L.rho;
  double ds[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) ds[k] = dm[k] - u[k] * dr;
  const double dsn = ds[0] * n[0] + ds[1] * n[1] + ds[2] * n[2];
  const double dpc = g.kappaM1 * ((R.E - L.E) - (u[0] * dm[0] + u[1] * dm[1] + (u[2] * dm[2] - q2 * dr)));
  const double ic2 = 0.5 * (ic * ic), a = c * dsn * ic2, b = dpc * ic2;
  const double w1 = 0.5 * l1 * (b - a), w5 = 0.5 * l5 * (b + a);
  const double h2 = 0.5 * l2, w2 = h2 * (dr - 2. * b);
  const double w15 = w1 + w5, W = w15 + w2, kn = (w5 - w1) * c - h2 * dsn;
  F[0] = F[0] - W;
#pragma unroll
  for (int k = 0; k < 3; ++k) F[1 + k] = F[1 + k] - (W * u[k] + (kn * n[k] + h2 * ds[k]));
  F[4] = F[4] - (w15 * H + (w2 * q2 + (kn * un + h2 * (u[0] * ds[0] + u[1] * ds[1] + u[2] * ds[2]))));
}

template <int RIEM, int CENTRAL, int PARAB>
__global__ void __launch_bounds__(128, 4)
k_face_dp(const double* __restrict__ Uf, const double* __restrict__ Pf, const double* __restrict__ Gf,
          const double* __restrict__ Fgeo, FaceGas gas, int nSides, int nBCSides, int n2, double* __restrict__ Flux) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x + (long long)nBCSides * n2;
  if (t >= (long long)nSides * n2) return;
  const int side = (int)(t / n2), pq = (int)(t - (long long)side * n2);
  const size_t S = nSides;
  const double* fg = Fgeo + (size_t)side * 10 * n2 + pq;
  const double n[3] = {fg[0], fg[n2], fg[2 * n2]};
  FaceSide L, R;
  auto load = [&](FaceSide& s, size_t slot) {
    const double* P = Pf + (slot * S + side) * 6 * n2 + pq;
    s.rho = P[0]; s.v[0] = P[n2]; s.v[1] = P[2 * n2]; s.v[2] = P[3 * n2]; s.p = P[4 * n2]; s.T = P[5 * n2];
    s.un = s.v[0] * n[0] + s.v[1] * n[1] + s.v[2] * n[2];
    s.E = Uf[((slot * S + side) * 5 + 4) * n2 + pq];
    s.srho = dp_rcp(s.rho);
  };
  load(L, 0);
  load(R, 1);
  double dm[3] = {0., 0., 0.}, F[5];
  if constexpr (RIEM != DG_RIEMANN_HLLC) {
    const double* m = Uf + (size_t)side * 5 * n2 + n2 + pq;
#pragma unroll
    for (int c = 0; c < 3; ++c) dm[c] = m[S * 5 * n2 + c * n2] - m[c * n2];
  }
  riemann_dp<RIEM, CENTRAL>(dm, L, R, n, gas, F);
  if constexpr (PARAB) {
    // F - mu/2 (t_L + t_R), t = (grad v + grad v^T - 2/3 div v) n; energy: v.t and lambda grad T.n
    double tq = 0., tv = 0., ts[3] = {0., 0., 0.};
#pragma unroll
    for (int slot = 0; slot < 2; ++slot) {
      const double* G = Gf + ((size_t)slot * S + side) * 15 * n2 + pq;
      const double ux = G[n2], vx = G[2 * n2], wx = G[3 * n2], Tx = G[4 * n2];
      const double uy = G[6 * n2], vy = G[7 * n2], wy = G[8 * n2], Ty = G[9 * n2];
      const double uz = G[11 * n2], vz = G[12 * n2], wz = G[13 * n2], Tz = G[14 * n2];
      const double d = (2. / 3.) * (ux + vy + wz);
      const double xy = uy + vx, xz = uz + wx, yz = vz + wy;
      const double t0 = fma(2., ux, -d) * n[0] + (xy * n[1] + xz * n[2]);
      const double t1 = xy * n[0] + (fma(2., vy, -d) * n[1] + yz * n[2]);
      const double t2 = xz * n[0] + (yz * n[1] + fma(2., wz, -d) * n[2]);
      const double* v = slot == 0 ? L.v : R.v;
      tv = fma(t0, v[0], fma(t1, v[1], fma(t2, v[2], tv)));
      tq = fma(Tx, n[0], fma(Ty, n[1], fma(Tz, n[2], tq)));
      if (slot == 0) { ts[0] = t0; ts[1] = t1; ts[2] = t2; }
      else { ts[0] = ts[0] + t0; ts[1] = ts[1] + t1; ts[2] = ts[2] + t2; }
    }
    const double hm = -0.5 * gas.mu;
#pragma unroll
    for (int c = 0; c < 3; ++c) F[1 + c] = fma(hm, ts[c], F[1 + c]);
    F[4] = fma(hm, tv, fma(-0.5 * gas.lambda, tq, F[4]));
  }
  const double se = fg[9 * n2];
  double* out = Flux + (size_t)side * 5 * n2 + pq;
#pragma unroll
  for (int v = 0; v < 5; ++v) out[v * n2] = F[v] * se;
}

}  // namespace gx

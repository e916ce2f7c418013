// Double-double numbers (Dekker's and Knuth's error-free sums and products) on the host, and the 1D basis in
// them: the fixed-point kernels hold its matrices with 58 to 62 bits, on every host the same.
#pragma once
#include <cmath>
#include <vector>

#include "../../include/galaexi_gb300.h"

namespace gxh {

struct DD {
  double h, l;
};
inline DD dd_add(DD a, DD b) {
  const double s = a.h + b.h, t = s - a.h;
  const double e = (a.h - (s - t)) + (b.h - t) + a.l + b.l;
  const double h = s + e;
  return {h, e - (h - s)};
}
inline DD dd_mul(DD a, DD b) {
  const double p = a.h * b.h;
  const double e = std::fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h);
  const double h = p + e;
  return {h, e - (h - p)};
}
inline DD dd_neg(DD a) { return {-a.h, -a.l}; }
inline DD dd_sub(DD a, DD b) { return dd_add(a, dd_neg(b)); }
inline DD dd_inv(DD a) {
  const double x = 1. / a.h;
  const DD r = dd_sub({1., 0.}, dd_mul(a, {x, 0.}));
  return dd_add({x, 0.}, {x * (r.h + r.l), 0.});
}
inline DD dd_num(double x) { return {x, 0.}; }
// a 2^bits, rounded
inline long long dd_fixed(DD a, int bits) { return std::llrint(std::ldexp(a.h, bits)) + std::llrint(std::ldexp(a.l, bits)); }

// nodes, quadrature weights, D(i,l) = l_l'(x_i) at [i n + l], l_i(1) = l_(N-i)(-1)
struct BasisDD {
  std::vector<DD> x, w, D, Lp;
};

// P_m and P_m' at x by the three-term recurrence
inline void dd_legendre(int m, DD x, DD& P, DD& dP) {
  DD p0 = dd_num(1.), p1 = x, d0 = dd_num(0.), d1 = dd_num(1.);
  for (int k = 2; k <= m; ++k) {
    const DD a = dd_mul(dd_num(2. * k - 1.), dd_inv(dd_num(k))), b = dd_mul(dd_num(k - 1.), dd_inv(dd_num(k)));
    const DD p2 = dd_sub(dd_mul(a, dd_mul(x, p1)), dd_mul(b, p0));
    const DD d2 = dd_add(d0, dd_mul(dd_num(2. * k - 1.), p1));
    p0 = p1; p1 = p2; d0 = d1; d1 = d2;
  }
  P = p1; dP = d1;
}

// x0: the FP64 nodes, refined here by Newton's iteration
inline void basis_dd(int N, int node_type, const std::vector<double>& x0, BasisDD& B) {
  const int n = N + 1;
  const bool gauss = node_type == DG_NODETYPE_GAUSS;
  B.x.assign(n, dd_num(0.)); B.w = B.x; B.Lp = B.x;
  B.D.assign((size_t)n * n, dd_num(0.));
  std::vector<DD> c(n);  // Gauss: P_n'(x_i); Gauss-Lobatto: P_N(x_i)
  for (int i = 0; i < n; ++i) {
    DD x = dd_num(x0[i]), P, dP;
    if (!gauss && (i == 0 || i == N)) x = dd_num(i == 0 ? -1. : 1.);
    else
      for (int it = 0; it < 3; ++it) {
        if (gauss) {  // zeros of P_n
          dd_legendre(n, x, P, dP);
          x = dd_sub(x, dd_mul(P, dd_inv(dP)));
        } else {  // zeros of P_N': (1 - x^2) P_N'' = 2 x P_N' - N (N+1) P_N
          dd_legendre(N, x, P, dP);
          const DD q = dd_sub(dd_num(1.), dd_mul(x, x));
          const DD d2 = dd_mul(dd_sub(dd_mul(dd_num(2.), dd_mul(x, dP)), dd_mul(dd_num(N * (N + 1.)), P)), dd_inv(q));
          x = dd_sub(x, dd_mul(dP, dd_inv(d2)));
        }
      }
    dd_legendre(gauss ? n : N, x, P, dP);
    const DD q = dd_sub(dd_num(1.), dd_mul(x, x));
    B.x[i] = x;
    if (gauss) {
      c[i] = dP;
      B.w[i] = dd_mul(dd_num(2.), dd_inv(dd_mul(q, dd_mul(dP, dP))));
      B.Lp[i] = dd_inv(dd_mul(dd_sub(dd_num(1.), x), dP));
      B.D[i * n + i] = dd_mul(x, dd_inv(q));
    } else {
      c[i] = P;
      B.w[i] = dd_mul(dd_num(2.), dd_inv(dd_mul(dd_num(N * (N + 1.)), dd_mul(P, P))));
      B.Lp[i] = dd_num(i == N ? 1. : 0.);
      B.D[i * n + i] = dd_num(i == 0 ? -N * (N + 1.) / 4. : (i == N ? N * (N + 1.) / 4. : 0.));
    }
  }
  for (int i = 0; i < n; ++i)
    for (int l = 0; l < n; ++l)
      if (l != i) B.D[i * n + l] = dd_mul(c[i], dd_inv(dd_mul(c[l], dd_sub(B.x[i], B.x[l]))));
}

}  // namespace gxh

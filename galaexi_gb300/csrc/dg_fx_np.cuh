// Launch code of the fixed-point kernels of the FP64 form for one compile-time node count NP = N+1.  Each
// dg_fx<NP>.cu includes this file with GX_NP defined.  They have translation units of their own: beside them
// the compiler laid the FP64 kernels of dg_np<NP>.cu out differently (prolongation at N = 5 up to 19% slower).
#pragma once
#include <cmath>
#include <cstring>
#include <vector>

#include "dg_ctx.h"
#include "dg_lift_fx.cuh"
#include "dg_lift_gfx.cuh"
#include "dg_volume_fx.cuh"
#include "dg_volume_wfx.cuh"

#ifndef GX_NP
#error "define GX_NP before including dg_fx_np.cuh"
#endif

namespace {

constexpr int NP = GX_NP;

#define GX_CUDA_TRY(call, what)                                                   \
  do {                                                                            \
    cudaError_t _e = (call);                                                      \
    if (_e != cudaSuccess) {                                                      \
      gxh::set_error(std::string(what) + ": " + cudaGetErrorString(_e));         \
      return DG_ERR_CUDA;                                                         \
    }                                                                             \
  } while (0)

template <typename K>
int smem_attr(K kern, size_t bytes, const char* what) {
  GX_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes), what);
  GX_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100), what);
  return DG_OK;
}

// the exponent e with |x| < 2^e for all entries of a matrix
int exponent(const std::vector<gxh::DD>& a) {
  double big = 0.;
  for (const gxh::DD& x : a) big = std::fabs(x.h) > big ? std::fabs(x.h) : big;
  int ex = 0;
  std::frexp(big * 1.01, &ex);
  return ex;
}
gx::FxDig digits(long long x) { return gx::FxDig{(int)(x >> 30), (int)(x & 0x3fffffff)}; }
gx::FxLimb limbs(long long x) {
  const int l = (int)(unsigned)(unsigned long long)x;
  return gx::FxLimb{(int)((x - l) / (1ll << 32)), l};
}

// a basis struct of a kernel, built once per context and kept there as bytes
template <typename B, typename F>
const B& kept(std::vector<unsigned char>& store, F build) {
  if (store.size() != sizeof(B)) {
    store.resize(sizeof(B));
    B b;
    std::memset(&b, 0, sizeof(B));
    build(b);
    std::memcpy(store.data(), &b, sizeof(B));
  }
  return *reinterpret_cast<const B*>(store.data());
}

// D_hat(i,l) = -w_l/w_i D(l,i) and L_hat(i) = L(i)/w_i in even and odd parts (VolWfxBasis).  A constant flux and
// its face fluxes cancel exactly: the diagonal even entry is what the others leave
void weak_basis(const dg_ctx* ctx, gx::VolWfxBasis<NP>& wb) {
  constexpr int N = NP - 1, H = gx::VolWfxBasis<NP>::H, HE = gx::VolWfxBasis<NP>::HE;
  const gxh::BasisDD& B = ctx->fxB;
  std::vector<gxh::DD> Dh(NP * NP), Lh(NP), all;
  for (int i = 0; i < NP; ++i) {
    const gxh::DD iw = gxh::dd_inv(B.w[i]);
    for (int l = 0; l < NP; ++l) Dh[i * NP + l] = gxh::dd_neg(gxh::dd_mul(gxh::dd_mul(B.w[l], iw), B.D[l * NP + i]));
    Lh[i] = gxh::dd_mul(B.Lp[i], iw);
  }
  all = Dh;
  all.insert(all.end(), Lh.begin(), Lh.end());
  wb.sD = 60 - exponent(all);
  double most = 0.;
  for (int i = 0; i < NP; ++i) {
    double sum = std::fabs(Lh[i].h) + std::fabs(Lh[N - i].h);
    for (int l = 0; l < NP; ++l) sum += std::fabs(Dh[i * NP + l].h);
    most = std::fmax(most, sum);
  }
  wb.S = (int)std::floor(63. - std::log2(3. * most) - 1e-3 - (59 + wb.sD - 64));
  auto half = [](gxh::DD a) { return gxh::dd_mul(a, gxh::dd_num(0.5)); };
  auto at = [&](int i, int l) { return Dh[i * NP + l]; };
  for (int i = 0; i < HE; ++i) {
    // L_hat_plus(i) = Lh[i], L_hat_minus(i) = Lh[N-i]
    const long long le = gxh::dd_fixed(half(gxh::dd_add(Lh[i], Lh[N - i])), wb.sD);
    const long long lo = gxh::dd_fixed(half(gxh::dd_sub(Lh[i], Lh[N - i])), wb.sD);
    wb.le[i] = limbs(le);
    long long rest = i < H ? lo : 0;
    if (i < H) wb.lo[i] = limbs(lo);
    for (int l = 0; l < HE; ++l) {
      if (i < H && l != i) {
        const long long ev = l < H ? gxh::dd_fixed(half(gxh::dd_add(at(i, l), at(i, N - l))), wb.sD)
                                   : gxh::dd_fixed(at(i, l), wb.sD - 1) * 2;
        rest += l < H ? ev : ev / 2;
        wb.even[i][l] = limbs(ev);
      }
      if (l < H) wb.odd[i][l] = limbs(gxh::dd_fixed(i < H ? half(gxh::dd_sub(at(i, l), at(i, N - l))) : at(i, l), wb.sD));
    }
    if (i < H) wb.even[i][i] = limbs(-rest);
  }
}

int volume_weak(dg_ctx* ctx, const double* U, const gx::Gas<double>& gas, gx::RKArgs rk, int rkmode, cudaStream_t st) {
  const gxc::PrecData<double>& P = ctx->d;
  const auto& wb = kept<gx::VolWfxBasis<NP>>(ctx->fx_weak, [&](gx::VolWfxBasis<NP>& b) { weak_basis(ctx, b); });
  auto kern = ctx->cfg.parabolic ? gx::k_volume_wfx<NP, 1> : gx::k_volume_wfx<NP, 0>;
  kern<<<ctx->nElems, gx::VolWfx<NP>::NT, gx::VolWfx<NP>::smem, st>>>(
      U, P.Pvol.p, P.Gvol.p, P.Met.p, ctx->MetL.p, P.Flux.p, ctx->E2S.p, wb, gxc::dev_basis(P, NP),
      ctx->cfg.node_type == DG_NODETYPE_GAUSS ? 1 : 0, gas, rk, rkmode);
  return DG_OK;
}

template <int SPL>
int volume_spl(dg_ctx* ctx, const double* U, const gx::Gas<double>& gas, gx::RKArgs rk, int rkmode, cudaStream_t st) {
  const gxc::PrecData<double>& P = ctx->d;
  auto kern = ctx->cfg.parabolic ? gx::k_volume_fx<NP, SPL, 1> : gx::k_volume_fx<NP, SPL, 0>;
  kern<<<ctx->nElems, gx::VolFx<NP>::NT, gx::VolFx<NP>::smem(ctx->cfg.parabolic), st>>>(
      U, P.Pvol.p, P.Gvol.p, P.Met.p, ctx->MetL.p, P.Flux.p, ctx->E2S.p,
      reinterpret_cast<const gx::VolFxBasis<NP>*>(ctx->fxb.p), gxc::dev_basis(P, NP), 1. / ctx->B.w[0], gas, rk, rkmode);
  return DG_OK;
}

int volume(dg_ctx* ctx, const double* U, const gx::Gas<double>& gas, gx::RKArgs rk, int rkmode, cudaStream_t st) {
  switch (ctx->cfg.split_dg) {
    case DG_SPLIT_NONE: return volume_weak(ctx, U, gas, rk, rkmode, st);
    case DG_SPLIT_KG: return volume_spl<DG_SPLIT_KG>(ctx, U, gas, rk, rkmode, st);
    default: return volume_spl<DG_SPLIT_PI>(ctx, U, gas, rk, rkmode, st);
  }
}

template <int SPL>
int configure_spl() {
  int rc = smem_attr(gx::k_volume_fx<NP, SPL, 0>, gx::VolFx<NP>::smem(0), "k_volume_fx attributes");
  return rc ? rc : smem_attr(gx::k_volume_fx<NP, SPL, 1>, gx::VolFx<NP>::smem(1), "k_volume_fx attributes");
}

// D in even and odd parts (LiftFxBasis).  The even parts of a row times (x_l + x_(N-l)) vanish exactly for a
// constant: the diagonal entry is what the others leave
void lift_basis(const dg_ctx* ctx, gx::LiftFxBasis<NP>& lb) {
  constexpr int N = NP - 1, H = gx::LiftFxBasis<NP>::H, HE = gx::LiftFxBasis<NP>::HE;
  const std::vector<gxh::DD>& D = ctx->fxB.D;
  lb.sD = 58 - exponent(D);
  auto at = [&](int i, int l) { return D[i * NP + l]; };
  auto half = [](gxh::DD a) { return gxh::dd_mul(a, gxh::dd_num(0.5)); };
  for (int i = 0; i < HE; ++i) {
    long long rest = 0;
    for (int l = 0; l < HE; ++l) {
      if (i < H && l != i) {
        const long long ev = l < H ? gxh::dd_fixed(half(gxh::dd_add(at(i, l), at(i, N - l))), lb.sD)
                                   : gxh::dd_fixed(at(i, l), lb.sD - 1) * 2;
        rest += l < H ? ev : ev / 2;
        lb.even[i][l] = digits(ev);
      }
      if (l < H)
        lb.odd[i][l] = digits(gxh::dd_fixed(i < H ? half(gxh::dd_sub(at(i, l), at(i, N - l))) : at(i, l), lb.sD));
    }
    if (i < H) lb.even[i][i] = digits(-rest);
  }
  lb.jump = digits(gxh::dd_fixed(gxh::dd_num(N * (N + 1) / 4.), lb.sD));
}

// the basis of k_lift_gfx (LiftGfxBasis)
void gauss_lift_basis(const dg_ctx* ctx, gx::LiftGfxBasis<NP>& gb) {
  constexpr int N = NP - 1, H = gx::LiftGfxBasis<NP>::H, HE = gx::LiftGfxBasis<NP>::HE;
  lift_basis(ctx, gb.d);
  const gxh::BasisDD& B = ctx->fxB;
  std::vector<gxh::DD> Lh(NP), LL(NP);
  for (int i = 0; i < NP; ++i) {
    Lh[i] = gxh::dd_mul(B.Lp[i], gxh::dd_inv(B.w[i]));
    LL[i] = gxh::dd_mul(gxh::dd_mul(B.Lp[i], Lh[i]), gxh::dd_num(ctx->cfg.eta_br2));
  }
  gb.sL = 58 - exponent(Lh);
  gb.sT = 58 - exponent(B.Lp);
  gxh::DD sum = gxh::dd_num(0.);
  for (const gxh::DD& x : LL) sum = gxh::dd_add(sum, x);
  gb.sLL = 59 - exponent({sum});  // (all of one sign)
  auto half = [](gxh::DD a) { return gxh::dd_mul(a, gxh::dd_num(0.5)); };
  for (int i = 0; i < NP; ++i) {
    gb.Lh[i] = digits(gxh::dd_fixed(Lh[i], gb.sL));
    gb.LL[i] = digits(gxh::dd_fixed(LL[i], gb.sLL));
  }
  for (int l = 0; l < HE; ++l) {
    gb.te[l] = digits(gxh::dd_fixed(l < H ? half(gxh::dd_add(B.Lp[l], B.Lp[N - l])) : B.Lp[l], gb.sT));
    if (l < H) gb.to[l] = digits(gxh::dd_fixed(half(gxh::dd_sub(B.Lp[l], B.Lp[N - l])), gb.sT));
  }
}

void lift_general(dg_ctx* ctx, cudaStream_t st) {
  gxc::PrecData<double>& P = ctx->d;
  const auto& gb = kept<gx::LiftGfxBasis<NP>>(ctx->fx_lift, [&](gx::LiftGfxBasis<NP>& b) { gauss_lift_basis(ctx, b); });
  const bool gauss = ctx->cfg.node_type == DG_NODETYPE_GAUSS, br2 = ctx->cfg.lifting == DG_LIFTING_BR2;
  auto kern = !gauss ? gx::k_lift_gfx<NP, false, true> : (br2 ? gx::k_lift_gfx<NP, true, true> : gx::k_lift_gfx<NP, true, false>);
  kern<<<ctx->nElems, gx::LiftGfx<NP>::NT, gx::LiftGfx<NP>::smem, st>>>(
      P.Pvol.p, P.Met.p, ctx->MetL.p, P.Pf.p, P.Fgeo.p, ctx->E2S.p, gb, gxc::dev_basis(P, NP), ctx->cfg.eta_br2,
      ctx->nSides, P.Gvol.p, P.Gf.p);
}

void lift(dg_ctx* ctx, cudaStream_t st) {
  if (ctx->cfg.node_type == DG_NODETYPE_GAUSS || ctx->cfg.lifting == DG_LIFTING_BR2) return lift_general(ctx, st);
  gxc::PrecData<double>& P = ctx->d;
  const auto& lb = kept<gx::LiftFxBasis<NP>>(ctx->fx_lift, [&](gx::LiftFxBasis<NP>& b) { lift_basis(ctx, b); });
  auto kern = ctx->face_exact ? gx::k_lift_fx<NP, true> : gx::k_lift_fx<NP, false>;
  kern<<<ctx->nElems, gx::LiftFx<NP>::NT, gx::LiftFx<NP>::smem, st>>>(
      P.Pvol.p, P.Met.p, ctx->MetL.p, P.Pf.p, P.Fgeo.p, ctx->E2S.p, lb, P.basis.p, ctx->B.Lhm[0], ctx->nSides, P.Gvol.p,
      P.Gf.p);
}

int configure(const dg_ctx* ctx) {
  const dg_config& c = ctx->cfg;
  int rc = DG_OK;
  if (c.split_dg == DG_SPLIT_NONE) {
    rc = smem_attr(gx::k_volume_wfx<NP, 0>, gx::VolWfx<NP>::smem, "k_volume_wfx attributes");
    if (rc == DG_OK) rc = smem_attr(gx::k_volume_wfx<NP, 1>, gx::VolWfx<NP>::smem, "k_volume_wfx attributes");
  }
  if (rc == DG_OK && c.parabolic) {
    const bool gauss = c.node_type == DG_NODETYPE_GAUSS, br2 = c.lifting == DG_LIFTING_BR2;
    if (!gauss && br2) rc = smem_attr(gx::k_lift_gfx<NP, false, true>, gx::LiftGfx<NP>::smem, "k_lift_gfx attributes");
    else if (br2) rc = smem_attr(gx::k_lift_gfx<NP, true, true>, gx::LiftGfx<NP>::smem, "k_lift_gfx attributes");
    else if (gauss) rc = smem_attr(gx::k_lift_gfx<NP, true, false>, gx::LiftGfx<NP>::smem, "k_lift_gfx attributes");
    else {
      rc = smem_attr(gx::k_lift_fx<NP, true>, gx::LiftFx<NP>::smem, "k_lift_fx attributes");
      if (rc == DG_OK) rc = smem_attr(gx::k_lift_fx<NP, false>, gx::LiftFx<NP>::smem, "k_lift_fx attributes");
    }
  }
  if (rc == DG_OK && c.split_dg == DG_SPLIT_PI) rc = configure_spl<DG_SPLIT_PI>();
  if (rc == DG_OK && c.split_dg == DG_SPLIT_KG) rc = configure_spl<DG_SPLIT_KG>();
  return rc;
}

}  // namespace

#define GX_CAT2(a, b) a##b
#define GX_CAT(a, b) GX_CAT2(a, b)
extern const gxc::FxTable GX_CAT(gx_fx_table_, GX_NP) = {configure, volume, lift};

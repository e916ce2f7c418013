// Launch code of the fixed-point kernels of the FP64 form for one compile-time node count NP = N+1.  Each
// dg_fx<NP>.cu includes this file with GX_NP defined.  They have translation units of their own: beside them
// the compiler laid the FP64 kernels of dg_np<NP>.cu out differently (prolongation at N = 5 up to 19% slower).
#pragma once
#include <cmath>

#include "dg_ctx.h"
#include "dg_lift_fx.cuh"
#include "dg_volume_fx.cuh"

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
  if constexpr (NP >= 3)
    return ctx->cfg.split_dg == DG_SPLIT_KG ? volume_spl<DG_SPLIT_KG>(ctx, U, gas, rk, rkmode, st)
                                            : volume_spl<DG_SPLIT_PI>(ctx, U, gas, rk, rkmode, st);
  gxh::set_error("split form needs N >= 2");
  return DG_ERR_UNSUPPORTED;
}

template <int SPL>
int configure_spl() {
  int rc = smem_attr(gx::k_volume_fx<NP, SPL, 0>, gx::VolFx<NP>::smem(0), "k_volume_fx attributes");
  return rc ? rc : smem_attr(gx::k_volume_fx<NP, SPL, 1>, gx::VolFx<NP>::smem(1), "k_volume_fx attributes");
}

// D of the Gauss-Lobatto nodes in even and odd parts (LiftFxBasis), from the basis limbs Q(i,l) 2^62 and
// w_0/w_i 2^60 of the context: D(i,l) = Q(i,l) / w_i = Q(i,l) (w_0/w_i) N(N+1)/2 off the diagonal, 0 on it but
// -+N(N+1)/4 at the ends
void lift_basis(const dg_ctx* ctx, gx::LiftFxBasis<NP>& lb) {
  constexpr int N = NP - 1, H = gx::LiftFxBasis<NP>::H, HE = gx::LiftFxBasis<NP>::HE;
  auto limb = [&](int at) { return (long long)ctx->fxh[2 * at] * (1ll << 32) + ctx->fxh[2 * at + 1]; };
  double big = 0.;
  for (int i = 0; i < NP; ++i)
    for (int l = 0; l < NP; ++l) big = std::fabs(ctx->B.D[i + NP * l]) > big ? std::fabs(ctx->B.D[i + NP * l]) : big;
  int ex = 0;
  std::frexp(big * 1.01, &ex);
  lb.sD = 58 - ex;
  auto D = [&](int i, int l) -> long long {  // D(i,l) 2^sD
    if (i == l) return i == 0 || i == N ? (i == 0 ? -1 : 1) * (long long)(((__int128)(N * (N + 1)) << lb.sD) / 4) : 0;
    const __int128 p = (__int128)limb(l + NP * i) * limb(NP * NP + i) / ((__int128)1 << 60);  // Q w_0/w_i 2^62
    return (long long)((p * (N * (N + 1) / 2)) / ((__int128)1 << (62 - lb.sD)));
  };
  auto dig = [](long long x) { return gx::FxDig{(int)(x >> 30), (int)(x & 0x3fffffff)}; };
  for (int i = 0; i < HE; ++i) {
    // the even parts of a row times (x_l + x_(N-l)) vanish exactly for a constant: the diagonal entry is what
    // the others leave
    long long rest = 0;
    for (int l = 0; l < HE; ++l) {
      long long ev = 0;
      if (i < H && l != i) {
        ev = l < H ? (D(i, l) + D(i, N - l)) / 2 : D(i, l) / 2 * 2;
        rest += l < H ? ev : ev / 2;
        lb.even[i][l] = dig(ev);
      }
      if (l < H) lb.odd[i][l] = dig(i < H ? (D(i, l) - D(i, N - l)) / 2 : D(i, l));
    }
    if (i < H) lb.even[i][i] = dig(-rest);
  }
  lb.jump = dig((long long)(((__int128)(N * (N + 1)) << lb.sD) / 4));
}

void lift(dg_ctx* ctx, cudaStream_t st) {
  if constexpr (NP >= 3) {
    gxc::PrecData<double>& P = ctx->d;
    gx::LiftFxBasis<NP> lb;
    lift_basis(ctx, lb);
    auto kern = ctx->face_exact ? gx::k_lift_fx<NP, true> : gx::k_lift_fx<NP, false>;
    kern<<<ctx->nElems, gx::LiftFx<NP>::NT, gx::LiftFx<NP>::smem, st>>>(
        P.Pvol.p, P.Met.p, ctx->MetL.p, P.Pf.p, P.Fgeo.p, ctx->E2S.p, lb, P.basis.p, ctx->B.Lhm[0], ctx->nSides, P.Gvol.p,
        P.Gf.p);
  }
}

int configure(const dg_ctx* ctx) {
  if constexpr (NP >= 3)
    if (ctx->cfg.parabolic && ctx->cfg.node_type == DG_NODETYPE_GAUSS_LOBATTO) {
      int rc = smem_attr(gx::k_lift_fx<NP, true>, gx::LiftFx<NP>::smem, "k_lift_fx attributes");
      if (rc == DG_OK) rc = smem_attr(gx::k_lift_fx<NP, false>, gx::LiftFx<NP>::smem, "k_lift_fx attributes");
      if (rc != DG_OK) return rc;
    }
  if constexpr (NP >= 3) {
    if (ctx->cfg.split_dg == DG_SPLIT_PI) return configure_spl<DG_SPLIT_PI>();
    if (ctx->cfg.split_dg == DG_SPLIT_KG) return configure_spl<DG_SPLIT_KG>();
  }
  return DG_OK;
}

}  // namespace

#define GX_CAT2(a, b) a##b
#define GX_CAT(a, b) GX_CAT2(a, b)
extern const gxc::FxTable GX_CAT(gx_fx_table_, GX_NP) = {configure, volume, lift};

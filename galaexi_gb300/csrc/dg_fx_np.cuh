// Launch code of the fixed-point kernels of the FP64 form for one compile-time node count NP = N+1.  Each
// dg_fx<NP>.cu includes this file with GX_NP defined.  They have translation units of their own: beside them
// the compiler laid the FP64 kernels of dg_np<NP>.cu out differently (prolongation at N = 5 up to 19% slower).
#pragma once
#include "dg_ctx.h"
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

int configure(const dg_ctx* ctx) {
  if constexpr (NP >= 3) {
    if (ctx->cfg.split_dg == DG_SPLIT_PI) return configure_spl<DG_SPLIT_PI>();
    if (ctx->cfg.split_dg == DG_SPLIT_KG) return configure_spl<DG_SPLIT_KG>();
  }
  return DG_OK;
}

}  // namespace

#define GX_CAT2(a, b) a##b
#define GX_CAT(a, b) GX_CAT2(a, b)
extern const gxc::FxTable GX_CAT(gx_fx_table_, GX_NP) = {configure, volume};

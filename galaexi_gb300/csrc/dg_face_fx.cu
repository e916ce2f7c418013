// Face kernels of the FP64 form (dg_face_fx.cuh), one per solver and central part.
#include "dg_ctx.h"
#include "dg_face_fx.cuh"

namespace {

template <int RIEM, int CENTRAL>
void launch(const dg_ctx* ctx, const gx::FaceGas& g, int n2, cudaStream_t st) {
  const gxc::PrecData<double>& P = ctx->d;
  const long long nt = (long long)(ctx->nSides - ctx->nBCSides) * n2;
  const int grid = (int)((nt + 127) / 128);
  if (ctx->cfg.parabolic)
    gx::k_face_dp<RIEM, CENTRAL, 1><<<grid, 128, 0, st>>>(P.Uf.p, P.Pf.p, P.Gf.p, P.Fgeo.p, g, ctx->nSides, ctx->nBCSides,
                                                          n2, P.Flux.p);
  else
    gx::k_face_dp<RIEM, CENTRAL, 0><<<grid, 128, 0, st>>>(P.Uf.p, P.Pf.p, P.Gf.p, P.Fgeo.p, g, ctx->nSides, ctx->nBCSides,
                                                          n2, P.Flux.p);
}
template <int RIEM>
bool by_central(const dg_ctx* ctx, const gx::FaceGas& g, int n2, cudaStream_t st) {
  switch (ctx->cfg.split_dg) {
    case DG_SPLIT_NONE: launch<RIEM, -1>(ctx, g, n2, st); return true;
    case DG_SPLIT_PI: launch<RIEM, DG_SPLIT_PI>(ctx, g, n2, st); return true;
    case DG_SPLIT_KG: launch<RIEM, DG_SPLIT_KG>(ctx, g, n2, st); return true;
  }
  return false;
}

}  // namespace

namespace gxc {

bool face_dp(const dg_ctx* ctx, const gx::Gas<double>& gas, cudaStream_t st) {
  const dg_config& c = ctx->cfg;
  const gx::FaceGas g{c.kappa - 1., c.kappa * c.R, gas.mu, gas.lambda};
  const int n2 = ctx->n2;
  switch (c.riemann) {
    case DG_RIEMANN_LF: return by_central<DG_RIEMANN_LF>(ctx, g, n2, st);
    case DG_RIEMANN_ROE: return by_central<DG_RIEMANN_ROE>(ctx, g, n2, st);
    case DG_RIEMANN_ROEENTROPYFIX: return by_central<DG_RIEMANN_ROEENTROPYFIX>(ctx, g, n2, st);
    case DG_RIEMANN_HLLC:
      if (c.split_dg != DG_SPLIT_NONE) return false;
      launch<DG_RIEMANN_HLLC, -1>(ctx, g, n2, st);
      return true;
  }
  return false;
}

}  // namespace gxc

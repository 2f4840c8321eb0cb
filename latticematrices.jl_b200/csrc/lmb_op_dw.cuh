// lmb_op_dw.cuh -- domain-wall (5D) operator policy and its field hooks.
#pragma once
#include "lmb_domainwall.cuh"
#include "lmb_domainwall_pair.cuh"
#include "lmb_driver.cuh"

namespace lmb {

// generalised / Mobius domain-wall operator on V4 * L5 sites
// (lmb_domainwall_set gives L5, mass, M, a, b, c)
struct DWPolicy {
  static constexpr int NC = 12;
  int prepare(lmb_ctx *ctx, int prec, cudaStream_t st) const {
    if (!ctx->geom_set) return fail(ctx, LMB_ERR_STATE, "lmb_set_geometry has not been called");
    if (!ctx->links[LMB_LINKS_THIN].valid) return fail(ctx, LMB_ERR_STATE, "gauge links have not been uploaded");
    if (ctx->dw_L5 <= 0) return fail(ctx, LMB_ERR_STATE, "lmb_domainwall_set has not been called");
    int rc = check_prec(ctx, prec);
    if (rc) return rc;
    return ensure_link_precision(ctx, ctx->links[LMB_LINKS_THIN], prec, st);
  }
  static bool one_pass(const lmb_ctx *ctx) { return ctx->dw_L5 <= kDslashThreads && !ctx->dw_two_pass; }
  // FP32 / int16: two slices per thread (every pair of slices is one 256-bit
  // word of a plane when L5 is even), where half as many threads still fill the
  // device.  Solves at L5 = 12 on 148 SMs by the blocks of pairs, one site ->
  // pairs, ms.
  // FP32, three blocks per SM (444 slots): from two thirds of the slots of its
  // waves on, so not between one wave and 1.33.  192 blocks 9.9 -> 10.3, 300 14.7
  // -> 14.0, 432 19.3 -> 17.0, 480 22.3 -> 24.1, 540 20.0 -> 21.8, 576 24.6 ->
  // 25.6, 630 25.8 -> 24.7, 864 33.7 -> 30.2, 945 35.9 -> 35.6, 1080 40.8 -> 40.0,
  // 1296 48.3 -> 44.3, 1728 70.1 -> 65.7.
  // int16, four (592): from 3/8 of them on, 222 blocks.  192 9.6 -> 9.8, 300 14.5
  // -> 13.8, 432 19.1 -> 17.1, 480 22.4 -> 21.8, 576 25.8 -> 21.7, 630 25.6 ->
  // 23.3, 864 32.5 -> 27.2, 1296 45.1 -> 39.8, 1728 65.2 -> 54.7.
  template <int P> static bool pairs(const lmb_ctx *ctx) {
    const int64_t threads = ctx->g.V * (ctx->dw_L5 / 2);
    constexpr int per_sm = DWPairBlocks<Field<P, 12>>::value;
    return one_pass(ctx) && ctx->pair_sites && ctx->adj_sites && ctx->dw_L5 % 2 == 0 &&
           (P == PREC_HALF ? fills_device(ctx, threads, per_sm, 3, 8) : fills_waves(ctx, threads, per_sm, 2, 3));
  }
  // the field between two passes (the two-pass launches, the small-lattice D5^+)
  template <int P> static bool make_tmp(lmb_ctx *ctx, Field<P, 12> &f) {
    return make_field(ctx, P == PREC_DOUBLE ? "dw_tmp_d" : (P == PREC_SINGLE ? "dw_tmp_s" : "dw_tmp_h"), f,
                      ctx->g.V * ctx->dw_L5);
  }
  // blocks of the largest launch (the one-pass adjoint holds whole 4D points)
  static int64_t max_blocks(const lmb_ctx *ctx) {
    const int64_t flat = grid_for(ctx->g.V * ctx->dw_L5, kDslashThreads);
    if (!one_pass(ctx)) return flat;
    const int64_t pts = grid_for(ctx->g.V, kDslashThreads / ctx->dw_L5);
    return pts > flat ? pts : flat;
  }
  DWParams params(const lmb_ctx *ctx) const {
    const int L5 = ctx->dw_L5;
    return DWParams{L5, ctx->dw_mass, ctx->dw_M, ctx->dw_coef, ctx->dw_coef + L5, ctx->dw_coef + 2 * L5};
  }
  template <int P, int DAG, class G, class Epi>
  int launch_g(lmb_ctx *ctx, const Field<P, 12> &in, const G &U, const Epi &epi, cudaStream_t st) const {
    typedef typename Real<P>::type R;
    const int64_t V4 = ctx->g.V, V5 = V4 * ctx->dw_L5;
    const DWParams d = params(ctx);
    const unsigned grid = grid_for(V5, kDslashThreads);
    if constexpr (P != PREC_DOUBLE) {
      if (pairs<P>(ctx)) {
        const int half = d.L5 / 2;
        if constexpr (!DAG) {
          dw_forward_pair_kernel<<<grid_for(V4 * half, kDslashThreads), kDslashThreads, 0, st>>>(ctx->g, in, U, d, epi);
        } else {
          const int npts = kDslashThreads / half;
          dw_adjoint_pair_kernel<<<grid_for(V4, npts), kDslashThreads, 0, st>>>(ctx->g, in, U, d, npts, epi);
        }
        LMB_CHECK_LAUNCH(ctx);
        return LMB_OK;
      }
    }
    if (one_pass(ctx)) {
      if constexpr (!DAG) {
        dw_forward_kernel<R><<<grid, kDslashThreads, 0, st>>>(ctx->g, in, U, d, epi);
      } else {
        const int npts = kDslashThreads / d.L5;
        dw_adjoint_kernel<R><<<grid_for(V4, npts), kDslashThreads, 0, st>>>(ctx->g, in, U, d, npts, epi);
      }
      LMB_CHECK_LAUNCH(ctx);
      return LMB_OK;
    }
    Field<P, 12> tmp;
    if (!make_tmp(ctx, tmp)) return fail(ctx, LMB_ERR_CUDA, "out of device memory (domain-wall workspace)");
    if constexpr (!DAG) {
      dw_fifth_kernel<P><<<grid, kDslashThreads, 0, st>>>(tmp, in, V4, d, epi);
      dw_stencil_kernel<R, 0, 1><<<grid, kDslashThreads, 0, st>>>(ctx->g, tmp, in, U, d, epi);
    } else {
      const EpiStoreFollow<P, Epi> e1{tmp, epi};
      dw_stencil_kernel<R, 1, 0><<<grid, kDslashThreads, 0, st>>>(ctx->g, in, in, U, d, e1);
      dw_adjoint_local_kernel<R><<<grid, kDslashThreads, 0, st>>>(in, tmp, V4, d, epi);
    }
    LMB_CHECK_LAUNCH(ctx);
    return LMB_OK;
  }
  template <int P, int DAG, class Epi>
  int launch(lmb_ctx *ctx, const Field<P, 12> &in, const Epi &epi, cudaStream_t st) const {
    const LinkSet &ls = ctx->links[LMB_LINKS_THIN];
    if (ls.recon(P)) return launch_g<P, DAG>(ctx, in, gauge12_view<P>(ls, ctx->g.V), epi, st);
    return launch_g<P, DAG>(ctx, in, gauge_view<P>(ls, ctx->g.V), epi, st);
  }
  int link_reals(const lmb_ctx *ctx, int prec) const { return ctx->links[LMB_LINKS_THIN].recon(prec) ? 12 : 18; }
  bool links_finite(const lmb_ctx *ctx) const { return ctx->links[LMB_LINKS_THIN].finite(); }
};

inline int64_t op_volume(const lmb_ctx *ctx, const DWPolicy &) { return ctx->g.V * ctx->dw_L5; }
template <> struct DirectOut<DWPolicy> { static constexpr bool value = true; };
inline int op_slices(const lmb_ctx *ctx, const DWPolicy &) { return ctx->dw_L5; }
inline int64_t op_max_blocks(const lmb_ctx *ctx, const DWPolicy &) { return DWPolicy::max_blocks(ctx); }
template <int PS> struct UsesRing<DWPolicy, PS> {
  static constexpr RingUse value = PS == PREC_DOUBLE ? RING_NEVER : RING_WHERE_IT_PAYS;
};
template <int PS> bool op_rings(const lmb_ctx *ctx, const DWPolicy &, int64_t bytes) {
  return bytes >= kRingBytes && DWPolicy::pairs<PS>(ctx);
}
template <int PS> bool op_reserve(lmb_ctx *ctx, const DWPolicy &) {
  Field<PS, 12> f;
  return DWPolicy::one_pass(ctx) || DWPolicy::make_tmp(ctx, f);
}
template <int PS, int NC>
int op_pack_in(lmb_ctx *ctx, const DWPolicy &, Field<PS, NC> &f, const void *src, cudaStream_t st) {
  const unsigned grid = grid_for(ctx->g.V * ctx->dw_L5, 256);
  if (ctx->dtype == LMB_DTYPE_C128)
    pack_field5_kernel<double2, PS, NC><<<grid, 256, 0, st>>>(f, (const double2 *)src, ctx->g, ctx->pd, ctx->dw_L5);
  else
    pack_field5_kernel<float2, PS, NC><<<grid, 256, 0, st>>>(f, (const float2 *)src, ctx->g, ctx->pd, ctx->dw_L5);
  LMB_CHECK_LAUNCH(ctx);
  return LMB_OK;
}
template <int PS, int NC>
int op_unpack_out(lmb_ctx *ctx, const DWPolicy &, void *dst, const Field<PS, NC> &f, cudaStream_t st) {
  const unsigned grid = grid_for(ctx->g.V * ctx->dw_L5, 256);
  if (ctx->dtype == LMB_DTYPE_C128)
    unpack_field5_kernel<double2, PS, NC><<<grid, 256, 0, st>>>((double2 *)dst, f, ctx->g, ctx->pd, ctx->dw_L5);
  else
    unpack_field5_kernel<float2, PS, NC><<<grid, 256, 0, st>>>((float2 *)dst, f, ctx->g, ctx->pd, ctx->dw_L5);
  LMB_CHECK_LAUNCH(ctx);
  return LMB_OK;
}

// small lattices (lmb_small_dw.cu)
template <int PS, int PX>
int op_cg_small(lmb_ctx *ctx, const DWPolicy &op, const Field<PS, 12> &p, const Field<PS, 12> &r,
                const Field<PS, 12> &t, const Field<PX, 12> &x, cudaStream_t st);

LMB_OP_INSTANCES(extern, DWPolicy)

}  // namespace lmb

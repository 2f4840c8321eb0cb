// lmb_small_wilson.cu -- Wilson / Wilson-clover instances of the small-lattice
// solver.
#include "lmb_op_wilson.cuh"
#include "lmb_small_host.cuh"

namespace lmb {

template <int PS, int PX, class G>
int small_wilson(lmb_ctx *ctx, const WilsonPolicy &op, const G &U, const Field<PS, 12> &p, const Field<PS, 12> &r,
                 const Field<PS, 12> &t, const Field<PX, 12> &x, cudaStream_t st) {
  typedef typename Real<PS>::type R;
  if (op.op == LMB_OP_WILSON_CLOVER)
    return small_cg(ctx,
                    SmallWilson<PS, G, Clover<PS>, true>{U, clover_view<PS>(ctx->clover, ctx->g.V), (R)op.kappa, {}}, p,
                    r, t, x, st);
  return small_cg(ctx, SmallWilson<PS, G, NoClover, false>{U, NoClover{ctx->g.V}, (R)op.kappa, {}}, p, r, t, x, st);
}

template <int PS, int PX>
int op_cg_small(lmb_ctx *ctx, const WilsonPolicy &op, const Field<PS, 12> &p, const Field<PS, 12> &r,
                const Field<PS, 12> &t, const Field<PX, 12> &x, cudaStream_t st) {
  if (!ctx->persistent) return kNotSmall;
  const LinkSet &ls = ctx->links[LMB_LINKS_THIN];
  if (ls.recon(PS)) return small_wilson<PS, PX>(ctx, op, gauge12_view<PS>(ls, ctx->g.V), p, r, t, x, st);
  return small_wilson<PS, PX>(ctx, op, gauge_view<PS>(ls, ctx->g.V), p, r, t, x, st);
}

#define LMB_SMALL_W(PS, PX)                                                                              \
  template int op_cg_small<PS, PX>(lmb_ctx *, const WilsonPolicy &, const Field<PS, 12> &,                \
                                   const Field<PS, 12> &, const Field<PS, 12> &, const Field<PX, 12> &, \
                                   cudaStream_t);
LMB_SMALL_W(PREC_DOUBLE, PREC_DOUBLE)
LMB_SMALL_W(PREC_SINGLE, PREC_SINGLE)
LMB_SMALL_W(PREC_HALF, PREC_SINGLE)

}  // namespace lmb

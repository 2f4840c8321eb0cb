// lmb_small_staggered.cu -- staggered / HISQ instances of the small-lattice
// solver.
#include "lmb_op_staggered.cuh"
#include "lmb_small_host.cuh"

namespace lmb {

template <int PS, int PX>
int op_cg_small(lmb_ctx *ctx, const StaggeredPolicy &op, const Field<PS, 3> &p, const Field<PS, 3> &r,
                const Field<PS, 3> &t, const Field<PX, 3> &x, cudaStream_t st) {
  typedef typename Real<PS>::type R;
  if (!ctx->persistent) return kNotSmall;
  const int64_t V = ctx->g.V;
  const R mass = (R)op.mass, fc = (R)0.5, lc = (R)(-(1.0 + op.eps) / 48.0);
  if (op.naik)
    return small_cg(ctx,
                    SmallStaggered<PS, Gauge<PS>, Gauge<PS>, true>{gauge_view<PS>(ctx->links[LMB_LINKS_FAT], V),
                                                                   gauge_view<PS>(ctx->links[LMB_LINKS_LONG], V), mass,
                                                                   fc, lc, {}},
                    p, r, t, x, st);
  const LinkSet &ls = ctx->links[LMB_LINKS_THIN];
  const NoLinks none{V};
  if (ls.recon(PS))
    return small_cg(ctx, SmallStaggered<PS, Gauge12<PS>, NoLinks, false>{gauge12_view<PS>(ls, V), none, mass, fc, lc, {}},
                    p, r, t, x, st);
  return small_cg(ctx, SmallStaggered<PS, Gauge<PS>, NoLinks, false>{gauge_view<PS>(ls, V), none, mass, fc, lc, {}}, p, r,
                  t, x, st);
}

#define LMB_SMALL_S(PS, PX)                                                                           \
  template int op_cg_small<PS, PX>(lmb_ctx *, const StaggeredPolicy &, const Field<PS, 3> &,           \
                                   const Field<PS, 3> &, const Field<PS, 3> &, const Field<PX, 3> &, \
                                   cudaStream_t);
LMB_SMALL_S(PREC_DOUBLE, PREC_DOUBLE)
LMB_SMALL_S(PREC_SINGLE, PREC_SINGLE)
LMB_SMALL_S(PREC_HALF, PREC_SINGLE)

}  // namespace lmb

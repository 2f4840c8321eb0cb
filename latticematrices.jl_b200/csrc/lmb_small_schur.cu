// lmb_small_schur.cu -- the even/odd Schur operator on small lattices
// (lmb_small.cuh): two passes per application, the odd sites' A^-1 H and the
// even sites' A - k^2 H, each on the V/2 sites of its parity.
#include "lmb_op_schur.cuh"
#include "lmb_small_host.cuh"

namespace lmb {

template <int PS, class G, bool CLOVER>
struct SmallSchur {
  static constexpr int NC = 12;
  typedef typename Real<PS>::type R;
  G U;                 // parity-ordered links and clover blocks
  Clover<PS> A, Ainv;
  R mk2;               // -kappa^2
  Field<PS, 12> mid;   // odd half field
  static constexpr int kWaves = 1;
  static constexpr int phases(int) { return 2; }
  LMB_HD int64_t sites(const Geom &g) const { return g.V / 2; }

  // E: dagger of the hops (the CG solves Dh Dh^+, so D of the driver is Dh^+)
  template <int E, int PAR, int W, class Src>
  LMB_D void hop_w(const Geom &g, int cb, const Src &f, SmallHops<R> &sm) const {
    constexpr int MU = W >> 1, BACK = W & 1;
    constexpr int PM = (E ? +1 : -1) * (BACK ? -1 : +1);
    int c[4], wrap;
    const int s = cb_site(g, cb, PAR, c);
    const int n = BACK ? bwd_site(g, s, c, MU, 1, &wrap) : fwd_site(g, s, c, MU, 1, &wrap);
    Cx<R> p[12], h[6], uh[6], u[9];
    f.load(n >> 1, p);
    U.load(MU, (BACK ? 1 - PAR : PAR) * (g.V / 2) + (BACK ? n >> 1 : cb), u);
    project<PM, MU>(p, h);
    if (wrap && ((g.phase_mask >> MU) & 1)) scale_phase(h, 6, BACK ? g.ph_bwd[MU] : g.ph_fwd[MU]);
    if (BACK) su3_adj_mul_half(u, h, uh);
    else su3_mul_half(u, h, uh);
    put_hop(sm, W, 6, uh);
  }
  template <int E, int PAR, class Src>
  LMB_D void hops(int w, const Geom &g, int cb, const Src &f, SmallHops<R> &sm) const {
    switch (w) {
      case 0: hop_w<E, PAR, 0>(g, cb, f, sm); break;
      case 1: hop_w<E, PAR, 1>(g, cb, f, sm); break;
      case 2: hop_w<E, PAR, 2>(g, cb, f, sm); break;
      case 3: hop_w<E, PAR, 3>(g, cb, f, sm); break;
      case 4: hop_w<E, PAR, 4>(g, cb, f, sm); break;
      case 5: hop_w<E, PAR, 5>(g, cb, f, sm); break;
      case 6: hop_w<E, PAR, 6>(g, cb, f, sm); break;
      default: hop_w<E, PAR, 7>(g, cb, f, sm); break;
    }
  }
  template <int DAG, int PH, class Src>
  LMB_D void hop(int w, const Geom &g, int cb, const Src &in, SmallHops<R> &sm) const {
    if constexpr (PH == 0) hops<1 - DAG, 1>(w, g, cb, in, sm);
    else hops<1 - DAG, 0>(w, g, cb, SrcField<PS, 12>{mid}, sm);
  }
  template <int E, int PH, int Q, class Src>
  LMB_D void spin(const Geom &g, int cb, const Src &in, const SmallHops<R> &sm, Cx<R> *out) const {
    constexpr int B = Q & 2;  // the clover block's first spin
    if constexpr (PH == 0) {
      if constexpr (CLOVER) {
        R a[36];
        Cx<R> v[6];
        Ainv.load(B >> 1, g.V / 2 + cb, a);
        sum_spin<E, B>(sm, v);
        sum_spin<E, B + 1>(sm, v + 3);
        herm6_rows<(Q & 1)>(a, v, out);
      } else {
        sum_spin<E, Q>(sm, out);
      }
    } else {
      Cx<R> acc[3], o[3];
      sum_spin<E, Q>(sm, acc);
      if constexpr (CLOVER) {
        R a[36];
        Cx<R> v[6];
        A.load(B >> 1, cb, a);
        in.own(cb, B, v);
        in.own(cb, B + 1, v + 3);
        herm6_rows<(Q & 1)>(a, v, o);
      } else {
        in.own(cb, Q, o);
      }
#pragma unroll
      for (int k = 0; k < 3; k++) out[k] = o[k] + mk2 * acc[k];
    }
  }
  template <int DAG, int PH, class Src>
  LMB_D void finish(int q, const Geom &g, int cb, const Src &in, const SmallHops<R> &sm, Cx<R> *out) const {
    switch (q) {
      case 0: spin<1 - DAG, PH, 0>(g, cb, in, sm, out); break;
      case 1: spin<1 - DAG, PH, 1>(g, cb, in, sm, out); break;
      case 2: spin<1 - DAG, PH, 2>(g, cb, in, sm, out); break;
      default: spin<1 - DAG, PH, 3>(g, cb, in, sm, out); break;
    }
  }
};

template <int PS, int PX, class G>
int small_schur(lmb_ctx *ctx, const SchurPolicy &op, const G &U, const Field<PS, 12> &p, const Field<PS, 12> &r,
                const Field<PS, 12> &t, const Field<PX, 12> &x, cudaStream_t st) {
  typedef typename Real<PS>::type R;
  Field<PS, 12> mid;
  if (!SchurPolicy::make_tmp(ctx, mid)) return kNotSmall;
  const Clover<PS> A = eo_clover_view<PS>(ctx, 0), Ai = eo_clover_view<PS>(ctx, 1);
  const R mk2 = (R)(-op.kappa * op.kappa);
  if (op.clover) return small_cg(ctx, SmallSchur<PS, G, true>{U, A, Ai, mk2, mid}, p, r, t, x, st);
  return small_cg(ctx, SmallSchur<PS, G, false>{U, A, Ai, mk2, mid}, p, r, t, x, st);
}

template <int PS, int PX>
int op_cg_small(lmb_ctx *ctx, const SchurPolicy &op, const Field<PS, 12> &p, const Field<PS, 12> &r,
                const Field<PS, 12> &t, const Field<PX, 12> &x, cudaStream_t st) {
  if (!ctx->persistent || ctx->dist) return kNotSmall;
  if (ctx->links[LMB_LINKS_THIN].recon(PS))
    return small_schur<PS, PX>(ctx, op, eo_gauge12_view<PS>(ctx), p, r, t, x, st);
  return small_schur<PS, PX>(ctx, op, eo_gauge_view<PS>(ctx), p, r, t, x, st);
}

#define LMB_SMALL_E(PS, PX)                                                                              \
  template int op_cg_small<PS, PX>(lmb_ctx *, const SchurPolicy &, const Field<PS, 12> &,                \
                                   const Field<PS, 12> &, const Field<PS, 12> &, const Field<PX, 12> &, \
                                   cudaStream_t);
LMB_SMALL_E(PREC_DOUBLE, PREC_DOUBLE)
LMB_SMALL_E(PREC_SINGLE, PREC_SINGLE)
LMB_SMALL_E(PREC_HALF, PREC_SINGLE)

}  // namespace lmb

// lmb_small_dw.cu -- the domain-wall operators on small lattices
// (lmb_small.cuh): D5 in one pass, D5^+ in two (Z = a D_W^+ psi to the
// intermediate field, then the local combination along the fifth dimension).
#include "lmb_op_dw.cuh"
#include "lmb_small_host.cuh"

namespace lmb {

template <int PS, class G>
struct SmallDW {
  static constexpr int NC = 12;
  typedef typename Real<PS>::type R;
  G U;
  DWParams d;
  Field<PS, 12> mid;  // Z
  static constexpr int kWaves = 1;
  static constexpr int phases(int dag) { return dag ? 2 : 1; }
  LMB_HD int64_t sites(const Geom &g) const { return g.V * d.L5; }

  template <int DAG, int W, class Src>
  LMB_D void hop_w(const Geom &g, int i, const Src &in, SmallHops<R> &sm) const {
    constexpr int MU = W >> 1, BACK = W & 1;
    constexpr int PM = (DAG ? +1 : -1) * (BACK ? -1 : +1);
    const int x4 = i / d.L5, s = i - x4 * d.L5;
    int c[4], wrap;
    site_coords(g, x4, c);
    const int n = BACK ? bwd_site(g, x4, c, MU, 1, &wrap) : fwd_site(g, x4, c, MU, 1, &wrap);
    Cx<R> p[12], h[6], uh[6], u[9];
    in.load(dw_idx(n, s, d.L5), p);
    U.load(MU, BACK ? n : x4, u);
    project<PM, MU>(p, h);
    if constexpr (!DAG) {  // of Y = b psi + c F psi (dw_Y_proj)
      int lo, hi;
      double flo, fhi;
      dw_F_sources(d, s, 0, lo, hi, flo, fhi);
      const R b = (R)d.b[s], cl = (R)d.c[s] * (R)flo, ch = (R)d.c[s] * (R)fhi;
      Cx<R> q[12], t[6];
      in.template part<0, 6>(dw_idx(n, lo, d.L5), q);
      in.template part<6, 12>(dw_idx(n, hi, d.L5), q);
      project_lower<PM, MU>(q, t);
#pragma unroll
      for (int k = 0; k < 6; k++) h[k] = b * h[k] + cl * q[k] + ch * t[k];
    }
    if (wrap && ((g.phase_mask >> MU) & 1)) scale_phase(h, 6, BACK ? g.ph_bwd[MU] : g.ph_fwd[MU]);
    if (BACK) su3_adj_mul_half(u, h, uh);
    else su3_mul_half(u, h, uh);
    put_hop(sm, W, 6, uh);
  }
  template <int DAG, int PH, class Src>
  LMB_D void hop(int w, const Geom &g, int i, const Src &in, SmallHops<R> &sm) const {
    if constexpr (PH == 0) {
      switch (w) {
        case 0: hop_w<DAG, 0>(g, i, in, sm); break;
        case 1: hop_w<DAG, 1>(g, i, in, sm); break;
        case 2: hop_w<DAG, 2>(g, i, in, sm); break;
        case 3: hop_w<DAG, 3>(g, i, in, sm); break;
        case 4: hop_w<DAG, 4>(g, i, in, sm); break;
        case 5: hop_w<DAG, 5>(g, i, in, sm); break;
        case 6: hop_w<DAG, 6>(g, i, in, sm); break;
        default: hop_w<DAG, 7>(g, i, in, sm); break;
      }
    }
  }
  template <int DAG, int PH, int Q, class Src>
  LMB_D void spin(int i, const Src &in, const SmallHops<R> &sm, Cx<R> *out) const {
    const int x4 = i / d.L5, s = i - x4 * d.L5;
    int lo, hi;
    double flo, fhi;
    dw_F_sources(d, s, DAG, lo, hi, flo, fhi);
    const int from = Q < 2 ? lo : hi;  // F's slice for this spin
    const double factor = Q < 2 ? flo : fhi;
    const R a = (R)d.a[s], diag = (R)(4.0 + d.M);
    Cx<R> p[3], f[3];
    in.own(i, Q, p);
    if constexpr (!DAG) {
      Cx<R> acc[3];
      sum_spin<0, Q>(sm, acc);
      in.own(dw_idx(x4, from, d.L5), Q, f);
      const R b = (R)d.b[s], c = (R)d.c[s];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const Cx<R> fk = (R)factor * f[k];
        const Cx<R> y = b * p[k] + c * fk;
        out[k] = a * (diag * y - (R)0.5 * acc[k] + p[k] - fk);
      }
    } else if constexpr (PH == 0) {
      Cx<R> acc[3];
      sum_spin<1, Q>(sm, acc);
#pragma unroll
      for (int k = 0; k < 3; k++) out[k] = a * (diag * p[k] - (R)0.5 * acc[k]);
    } else {
      Cx<R> z[3], zn[3];
      const int64_t n = dw_idx(x4, from, d.L5);
      in.own(n, Q, f);
      own_load(mid, i, Q, z);
      own_load(mid, n, Q, zn);
      const R b = (R)d.b[s], pf = (R)(factor * d.a[from]), zf = (R)(factor * d.c[from]);
#pragma unroll
      for (int k = 0; k < 3; k++) out[k] = a * p[k] - pf * f[k] + b * z[k] + zf * zn[k];
    }
  }
  template <int DAG, int PH, class Src>
  LMB_D void finish(int q, const Geom &, int i, const Src &in, const SmallHops<R> &sm, Cx<R> *out) const {
    switch (q) {
      case 0: spin<DAG, PH, 0>(i, in, sm, out); break;
      case 1: spin<DAG, PH, 1>(i, in, sm, out); break;
      case 2: spin<DAG, PH, 2>(i, in, sm, out); break;
      default: spin<DAG, PH, 3>(i, in, sm, out); break;
    }
  }
};

template <int PS, int PX>
int op_cg_small(lmb_ctx *ctx, const DWPolicy &op, const Field<PS, 12> &p, const Field<PS, 12> &r,
                const Field<PS, 12> &t, const Field<PX, 12> &x, cudaStream_t st) {
  if (!ctx->persistent) return kNotSmall;
  Field<PS, 12> mid;
  if (!DWPolicy::make_tmp(ctx, mid)) return kNotSmall;
  const DWParams d = op.params(ctx);
  const LinkSet &ls = ctx->links[LMB_LINKS_THIN];
  if (ls.recon(PS))
    return small_cg(ctx, SmallDW<PS, Gauge12<PS>>{gauge12_view<PS>(ls, ctx->g.V), d, mid}, p, r, t, x, st);
  return small_cg(ctx, SmallDW<PS, Gauge<PS>>{gauge_view<PS>(ls, ctx->g.V), d, mid}, p, r, t, x, st);
}

#define LMB_SMALL_D(PS, PX)                                                                           \
  template int op_cg_small<PS, PX>(lmb_ctx *, const DWPolicy &, const Field<PS, 12> &,                \
                                   const Field<PS, 12> &, const Field<PS, 12> &, const Field<PX, 12> &, \
                                   cudaStream_t);
LMB_SMALL_D(PREC_DOUBLE, PREC_DOUBLE)
LMB_SMALL_D(PREC_SINGLE, PREC_SINGLE)
LMB_SMALL_D(PREC_HALF, PREC_SINGLE)

}  // namespace lmb

// lmb_force_ops.cu -- HISQ smearing chain (Fat7 / Lepage, U(3) projection,
// Naik), the HISQ and Wilson-clover link pullbacks and fermion forces.
#include "lmb_clover_force.cuh"
#include "lmb_fat7.cuh"
#include "lmb_hisq_force.cuh"
#include "lmb_op_staggered.cuh"
#include "lmb_op_wilson.cuh"

using namespace lmb;

namespace lmb {

// extent of a block of sites along an axis of n sites: the one of `most`, most
// - 1, .. (most + 1) / 2 that leaves the fewest idle lanes in the last block
int block_extent(int n, int most) {
  if (n <= most) return n;
  int best = most;
  for (int t = most - 1; 2 * t > most; t--)
    if ((n + t - 1) / t * t < (n + best - 1) / best * best) best = t;
  return best;
}
// A block of up to kFat7Threads sites, long first in x (whole lines of eight
// sites), then along the axes of `order` in turn: those along which the
// kernel's matrices are read again by the neighbour.  With four sites along
// both axes of a transport, half of its six gathered matrices hit L1.
SiteTile fat7_tile(const Geom &g, const int *order, int norder) {
  SiteTile t{{1, 1, 1, 1}, {0, 0, 0, 0}};
  t.t[0] = block_extent(g.L[0], 8);
  int left = kFat7Threads / t.t[0];
  for (int pass = 0; pass < 2; pass++)
    for (int i = 0; i < norder; i++) {
      const int d = order[i];
      if (d == 0) continue;
      const int now = t.t[d];
      const int most = std::min(pass ? 8 : 4, left * now);
      if (most <= now) continue;
      t.t[d] = std::max(now, block_extent(g.L[d], most));
      left = left * now / t.t[d];
    }
  for (int d = 0; d < 4; d++) t.n[d] = (g.L[d] + t.t[d] - 1) / t.t[d];
  return t;
}
unsigned blocks_of(const SiteTile &t) { return (unsigned)t.n[0] * t.n[1] * t.n[2] * t.n[3]; }

// fields of nine planes a Fat7 map keeps per direction: S and M (M+ and M- with
// the Lepage term) of the three axes, for the gradient twice
int64_t fat7_fields(bool lepage, bool gradient) { return (lepage ? 9 : 6) * (gradient ? 2 : 1); }

struct Fat7Launch {
  int nmu;         // directions per launch
  int64_t per_mu;  // stride of their workspaces
  double2 *work;   // nullptr: out of memory
};
// Directions per launch.  One direction's three axes give V / 128 x 3 blocks;
// below 64 Ki sites that is less than about four waves of the 148 SMs, and
// the four directions share a launch (their workspaces then hold at most
// 700 MB).  Larger lattices, and those whose four workspaces find no memory,
// keep one direction's.  `fields`: of the largest map of the call, which asks
// once, so that no level's workspace is freed for the next one's.
Fat7Launch fat7_launch(lmb_ctx *ctx, int64_t fields) {
  const int64_t per_mu = fields * 9 * ctx->g.V;
  const size_t bytes = sizeof(double2) * per_mu;
  double2 *work = ctx->g.V <= (1 << 16) ? (double2 *)spare_workspace(ctx, "fat7", 4 * bytes) : nullptr;
  if (work) return Fat7Launch{4, per_mu, work};
  return Fat7Launch{1, per_mu, (double2 *)workspace(ctx, "fat7", bytes)};
}

// block shapes of a stage for the directions mu0 .. mu0 + nmu - 1, and the
// largest number of blocks
enum Fat7Stage { F7_THREE, F7_FIVE, F7_SUM, F7_GRAD };
unsigned fat7_tiles(const Geom &g, Fat7Stage stage, int mu0, int nmu, Fat7Tiles &tl) {
  unsigned most = 0;
  for (int i = 0; i < nmu; i++)
    for (int slot = 0; slot < 3; slot++) {
      const int mu = mu0 + i;
      int ax[3], k = 0;
      for (int d = 0; d < 4; d++)
        if (d != mu) ax[k++] = d;
      const int a = slot == 0 ? 1 : 0, c = slot == 2 ? 1 : 2;
      const int three[4] = {ax[slot], mu, ax[a], ax[c]}, five[4] = {ax[a], ax[c], mu, ax[slot]};
      const int sum[4] = {mu, ax[0], ax[1], ax[2]}, grad[4] = {mu, ax[2], ax[1], ax[0]};
      const int *order = stage == F7_THREE ? three : stage == F7_FIVE ? five : stage == F7_SUM ? sum : grad;
      tl.t[i][slot] = fat7_tile(g, order, 4);
      most = std::max(most, blocks_of(tl.t[i][slot]));
    }
  return most;
}

template <int NF, bool LEPAGE>
void fat7_staples(lmb_ctx *ctx, const Fat7Launch &l, const double2 *U, const Fat7Field &f0, const Fat7Field &f1,
                  int mu0, const double *coef, cudaStream_t st) {
  Fat7Tiles tl;
  unsigned n = fat7_tiles(ctx->g, F7_THREE, mu0, l.nmu, tl);
  fat7_three_kernel<NF, LEPAGE><<<dim3(3 * n, l.nmu), kFat7Threads, 0, st>>>(ctx->g, tl, U, f0, f1, mu0, l.per_mu);
  n = fat7_tiles(ctx->g, F7_FIVE, mu0, l.nmu, tl);
  fat7_five_kernel<NF, LEPAGE><<<dim3(3 * n, l.nmu), kFat7Threads, 0, st>>>(ctx->g, tl, U, f0, f1, mu0, l.per_mu,
                                                                            coef[2], coef[3], coef[4]);
}

template <bool ACCUMULATE>
void fat7_sum(lmb_ctx *ctx, const Fat7Launch &l, const double2 *U, double2 *out, const Fat7Field &f, int mu0,
              double c1, cudaStream_t st) {
  Fat7Tiles tl;
  const unsigned n = fat7_tiles(ctx->g, F7_SUM, mu0, l.nmu, tl);
  fat7_sum_kernel<ACCUMULATE><<<dim3(n, l.nmu), kFat7Threads, 0, st>>>(ctx->g, tl, U, out, f, mu0, l.per_mu, c1);
}

// V = Fat7(U) with coefficients (c1, c3, c5, c7, cLepage)
int fat7_planes(lmb_ctx *ctx, const Fat7Launch &l, const double2 *U, double2 *V, const double *coef,
                cudaStream_t st) {
  const int64_t F3 = 27 * ctx->g.V;  // the three axes' fields
  const bool lepage = coef[4] != 0.0;
  double2 *work = l.work;
  const Fat7Field f{U, work, work + F3, lepage ? work + 2 * F3 : work + F3, coef[1]};
  for (int mu = 0; mu < 4; mu += l.nmu) {
    if (lepage)
      fat7_staples<1, true>(ctx, l, U, f, f, mu, coef, st);
    else
      fat7_staples<1, false>(ctx, l, U, f, f, mu, coef, st);
    fat7_sum<false>(ctx, l, U, V, f, mu, coef[0], st);
  }
  LMB_CHECK_LAUNCH(ctx);
  return LMB_OK;
}

int project_u3_planes(lmb_ctx *ctx, const double2 *V, double2 *W, cudaStream_t st) {
  u3_project_kernel<<<grid_for(4 * ctx->g.V, kSmearThreads), kSmearThreads, 0, st>>>(W, V, ctx->g.V);
  LMB_CHECK_LAUNCH(ctx);
  return LMB_OK;
}

int naik_planes(lmb_ctx *ctx, const double2 *W, double2 *L, cudaStream_t st) {
  naik_kernel<<<grid_for(4 * ctx->g.V, kSmearThreads), kSmearThreads, 0, st>>>(L, W, ctx->g);
  LMB_CHECK_LAUNCH(ctx);
  return LMB_OK;
}

// storage of a derived (not uploaded) link set, to be written in place and
// then installed
double2 *derived_planes(lmb_ctx *ctx, int which) {
  LinkSet &ls = ctx->links[which];
  ls.valid = false;
  if (!ls.d && device_malloc(ctx, &ls.d, sizeof(double2) * 36 * ctx->g.V) != cudaSuccess) ls.d = nullptr;
  return ls.d;
}
int install_links(lmb_ctx *ctx, int which, cudaStream_t st) {
  LinkSet &ls = ctx->links[which];
  int rc;
  ls.scale = device_absmax(ctx, ls.d, 36 * ctx->g.V, st, &rc);
  if (rc) return rc;
  ls.su3_dev = 1.0;  // smeared links are not SU(3): never reconstruct
  for (int mu = 0; mu < 4; mu++) {
    ls.ptr[mu] = nullptr;
    ls.epoch[mu] = 0;
  }
  ls.valid = true;
  ls.version++;
  return LMB_OK;
}

// dU += d/dU Re<dV, Fat7(U)>: the staples of U and of dV, the Fat7 map of dV
// onto its own direction, and the transports' links
int fat7_pullback_planes(lmb_ctx *ctx, const Fat7Launch &l, const double2 *U, const double2 *dV, double2 *dU,
                         const double *coef, cudaStream_t st) {
  const int64_t F3 = 27 * ctx->g.V;
  const bool lepage = coef[4] != 0.0;
  double2 *work = l.work;
  const Fat7Field fu{U, work, work + F3, lepage ? work + 4 * F3 : work + F3, 0.0};
  const Fat7Field fg{dV, work + 2 * F3, work + 3 * F3, lepage ? work + 5 * F3 : work + 3 * F3, coef[1]};
  for (int mu = 0; mu < 4; mu += l.nmu) {
    if (lepage)
      fat7_staples<2, true>(ctx, l, U, fu, fg, mu, coef, st);
    else
      fat7_staples<2, false>(ctx, l, U, fu, fg, mu, coef, st);
    fat7_sum<true>(ctx, l, U, dU, fg, mu, coef[0], st);
    Fat7Tiles tl;
    const unsigned n = fat7_tiles(ctx->g, F7_GRAD, mu, 1, tl);
    fat7_grad_kernel<<<4 * n, kFat7Threads, 0, st>>>(ctx->g, tl, U, dU, fu, fg, mu, l.nmu, l.per_mu, coef[3]);
  }
  LMB_CHECK_LAUNCH(ctx);
  return LMB_OK;
}

// dU_planes += d/dU [coef Re<dr, D_HISQ(U) psi>] through the whole chain
int hisq_pullback_planes(lmb_ctx *ctx, const double2 *thin, const Field<PREC_DOUBLE, 3> &dr,
                         const Field<PREC_DOUBLE, 3> &psi, double naik_epsilon, double coefficient, double2 *dU,
                         cudaStream_t st) {
  const int64_t n = ctx->g.V;
  const size_t L36 = sizeof(double2) * 36 * n;
  double2 *V1 = (double2 *)workspace(ctx, "force_V1", L36), *W = (double2 *)workspace(ctx, "force_W", L36);
  double2 *dX = (double2 *)workspace(ctx, "force_dX", L36), *dL = (double2 *)workspace(ctx, "force_dL", L36);
  double2 *dW = (double2 *)workspace(ctx, "force_dW", L36), *dV1 = (double2 *)workspace(ctx, "force_dV1", L36);
  if (!V1 || !W || !dX || !dL || !dW || !dV1) return fail(ctx, LMB_ERR_CUDA, "out of device memory (force)");
  const double c_level1[5] = {1.0 / 8, 1.0 / 16, 1.0 / 64, 1.0 / 384, 0.0};
  const double c_level2[5] = {1.0 + naik_epsilon / 8, 1.0 / 16, 1.0 / 64, 1.0 / 384, -1.0 / 8};
  int rc;
  const Fat7Launch l = fat7_launch(ctx, fat7_fields(true, true));
  if (!l.work) return fail(ctx, LMB_ERR_CUDA, "out of device memory (force staples)");
  // recompute the smearing levels the pullback needs
  if ((rc = fat7_planes(ctx, l, thin, V1, c_level1, st))) return rc;
  if ((rc = project_u3_planes(ctx, V1, W, st))) return rc;
  // Dirac outer products
  const double fc = coefficient / 2, lc = -coefficient * (1.0 + naik_epsilon) / 48.0;
  hisq_outer_product_kernel<<<grid_for(n, kSmearThreads), kSmearThreads, 0, st>>>(dX, dL, dr, psi, ctx->g, fc, lc);
  LMB_CHECK_LAUNCH(ctx);
  // Naik and level-2 Fat7 -> dW
  LMB_CUDA(ctx, cudaMemsetAsync(dW, 0, L36, st));
  naik_pullback_kernel<<<grid_for(4 * n, kSmearThreads), kSmearThreads, 0, st>>>(dW, dL, W, ctx->g);
  LMB_CHECK_LAUNCH(ctx);
  if ((rc = fat7_pullback_planes(ctx, l, W, dX, dW, c_level2, st))) return rc;
  // U(3) projection -> dV1
  LMB_CUDA(ctx, cudaMemsetAsync(dV1, 0, L36, st));
  u3_pullback_kernel<<<grid_for(4 * n, 64), 64, 0, st>>>(dV1, dW, V1, n);
  LMB_CHECK_LAUNCH(ctx);
  // level-1 Fat7 -> thin links
  return fat7_pullback_planes(ctx, l, thin, dV1, dU, c_level1, st);
}

// grad (36 planes) = d/dU [coef Re<dr, D_clover(U) psi>]
int clover_pullback_planes(lmb_ctx *ctx, const double2 *thin, const Field<PREC_DOUBLE, 12> &dr,
                           const Field<PREC_DOUBLE, 12> &psi, double kappa, double csw, double coefficient,
                           double2 *grad, cudaStream_t st) {
  const int64_t n = ctx->g.V;
  wilson_outer_product_kernel<<<grid_for(n, 128), 128, 0, st>>>(grad, dr, psi, ctx->g, -kappa * coefficient);
  LMB_CHECK_LAUNCH(ctx);
  if (csw == 0.0) return LMB_OK;
  // the packed H of the six planes and the inserted links of all of them at once
  // (1728 B per site), or of one plane at a time on lattices above 4 Mi sites and
  // where those of six find no memory: together less than the six full cotangents.
  // One workspace: an allocation takes 0.3 ms of a first call
  const int64_t plane = 18 * n, packed = 6 * kAntiPlanes * n;
  double2 *H = nullptr;
  if (n <= (1 << 22)) H = (double2 *)spare_workspace(ctx, "force_clover", sizeof(double2) * (packed + 6 * plane));
  const int np = H ? 6 : 1;
  if (!H) H = (double2 *)workspace(ctx, "force_clover", sizeof(double2) * (packed + plane));
  if (!H) return fail(ctx, LMB_ERR_CUDA, "out of device memory (clover force)");
  double2 *W = H + packed;
  clover_cotangent_kernel<<<grid_for(n, 128), 128, 0, st>>>(H, dr, psi, ctx->g, -kappa * csw * coefficient);
  LMB_CHECK_LAUNCH(ctx);
  Fat7Tiles tl;
  const unsigned blocks = fat7_tiles(ctx->g, F7_SUM, 0, 4, tl);
  for (int p = 0; p < 6; p += np) {
    clover_insert_kernel<<<dim3(grid_for(n, kFat7Threads), 2 * np), kFat7Threads, 0, st>>>(W, thin, H, ctx->g, p);
    clover_link_pullback_kernel<<<4 * blocks, kFat7Threads, 0, st>>>(grad, thin, W, ctx->g, tl, p, np);
    LMB_CHECK_LAUNCH(ctx);
  }
  return LMB_OK;
}

int accumulate_links_to(lmb_ctx *ctx, void *const dU[4], const double2 *planes, cudaStream_t st) {
  const unsigned grid = grid_for(ctx->g.V, kSmearThreads);
  if (ctx->dtype == LMB_DTYPE_C128)
    accumulate_links_kernel<double2><<<grid, kSmearThreads, 0, st>>>((double2 *)dU[0], (double2 *)dU[1], (double2 *)dU[2],
                                                            (double2 *)dU[3], planes, ctx->g, ctx->pd);
  else
    accumulate_links_kernel<float2><<<grid, kSmearThreads, 0, st>>>((float2 *)dU[0], (float2 *)dU[1], (float2 *)dU[2],
                                                           (float2 *)dU[3], planes, ctx->g, ctx->pd);
  LMB_CHECK_LAUNCH(ctx);
  return LMB_OK;
}


}  // namespace lmb

extern "C" {

int lmb_hisq_fat7(lmb_ctx *ctx, const void *const U[4], const double coefficients[5], void *const V[4],
                  void *stream) {
  if (!ctx_ok(ctx)) return LMB_ERR_ARG;
  if (!ctx->geom_set) return fail(ctx, LMB_ERR_STATE, "lmb_set_geometry has not been called");
  int rc = check_links_arg(ctx, U, "input link");
  if (rc) return rc;
  if ((rc = check_links_arg(ctx, (const void *const *)V, "output link"))) return rc;
  if (!coefficients) return fail(ctx, LMB_ERR_ARG, "null coefficients");
  cudaStream_t st = as_stream(stream);
  const int64_t n = ctx->g.V;
  double2 *in = (double2 *)workspace(ctx, "smear_in", sizeof(double2) * 36 * n);
  double2 *out = (double2 *)workspace(ctx, "smear_out", sizeof(double2) * 36 * n);
  if (!in || !out) return fail(ctx, LMB_ERR_CUDA, "out of device memory (smearing)");
  const Fat7Launch l = fat7_launch(ctx, fat7_fields(coefficients[4] != 0.0, false));
  if (!l.work) return fail(ctx, LMB_ERR_CUDA, "out of device memory (smearing staples)");
  if ((rc = pack_links_to(ctx, in, U, st))) return rc;
  if ((rc = fat7_planes(ctx, l, in, out, coefficients, st))) return rc;
  return unpack_links_from(ctx, V, out, st);
}

int lmb_hisq_project_u3(lmb_ctx *ctx, const void *const V[4], void *const W[4], void *stream) {
  if (!ctx_ok(ctx)) return LMB_ERR_ARG;
  if (!ctx->geom_set) return fail(ctx, LMB_ERR_STATE, "lmb_set_geometry has not been called");
  int rc = check_links_arg(ctx, V, "input link");
  if (rc) return rc;
  if ((rc = check_links_arg(ctx, (const void *const *)W, "output link"))) return rc;
  cudaStream_t st = as_stream(stream);
  const int64_t n = ctx->g.V;
  double2 *in = (double2 *)workspace(ctx, "smear_in", sizeof(double2) * 36 * n);
  double2 *out = (double2 *)workspace(ctx, "smear_out", sizeof(double2) * 36 * n);
  if (!in || !out) return fail(ctx, LMB_ERR_CUDA, "out of device memory (smearing)");
  if ((rc = pack_links_to(ctx, in, V, st))) return rc;
  if ((rc = project_u3_planes(ctx, in, out, st))) return rc;
  return unpack_links_from(ctx, W, out, st);
}

int lmb_hisq_naik(lmb_ctx *ctx, const void *const W[4], void *const L[4], void *stream) {
  if (!ctx_ok(ctx)) return LMB_ERR_ARG;
  if (!ctx->geom_set) return fail(ctx, LMB_ERR_STATE, "lmb_set_geometry has not been called");
  int rc = check_links_arg(ctx, W, "input link");
  if (rc) return rc;
  if ((rc = check_links_arg(ctx, (const void *const *)L, "output link"))) return rc;
  cudaStream_t st = as_stream(stream);
  const int64_t n = ctx->g.V;
  double2 *in = (double2 *)workspace(ctx, "smear_in", sizeof(double2) * 36 * n);
  double2 *out = (double2 *)workspace(ctx, "smear_out", sizeof(double2) * 36 * n);
  if (!in || !out) return fail(ctx, LMB_ERR_CUDA, "out of device memory (smearing)");
  if ((rc = pack_links_to(ctx, in, W, st))) return rc;
  if ((rc = naik_planes(ctx, in, out, st))) return rc;
  return unpack_links_from(ctx, L, out, st);
}

int lmb_hisq_links_from_thin(lmb_ctx *ctx, const void *const U[4], const uint64_t epoch[4], double naik_epsilon,
                             void *const X[4], void *const L[4], void *stream) {
  if (!ctx_ok(ctx)) return LMB_ERR_ARG;
  if (!ctx->geom_set) return fail(ctx, LMB_ERR_STATE, "lmb_set_geometry has not been called");
  int rc = check_links_arg(ctx, U, "thin link");
  if (rc) return rc;
  if (!std::isfinite(naik_epsilon)) return fail(ctx, LMB_ERR_ARG, "naik_epsilon must be finite");
  cudaStream_t st = as_stream(stream);
  lmb_smear_key &key = ctx->smear;
  bool same = key.valid && key.naik_epsilon == naik_epsilon && ctx->links[LMB_LINKS_FAT].valid &&
              ctx->links[LMB_LINKS_LONG].valid && epoch;
  for (int mu = 0; mu < 4 && same; mu++) same = key.ptr[mu] == U[mu] && key.epoch[mu] == epoch[mu];
  const int64_t n = ctx->g.V;
  if (!same) {
    double2 *thin = (double2 *)workspace(ctx, "smear_thin", sizeof(double2) * 36 * n);
    double2 *w = (double2 *)workspace(ctx, "smear_w", sizeof(double2) * 36 * n);
    key.valid = false;  // the link sets are rewritten in place
    double2 *fat = derived_planes(ctx, LMB_LINKS_FAT), *lng = derived_planes(ctx, LMB_LINKS_LONG);
    if (!thin || !w || !fat || !lng) return fail(ctx, LMB_ERR_CUDA, "out of device memory (smearing)");
    // hisq_links_from_thin! (HISQFullSmearing.jl:284-293)
    const double c_level1[5] = {1.0 / 8, 1.0 / 16, 1.0 / 64, 1.0 / 384, 0.0};
    const double c_level2[5] = {1.0 + naik_epsilon / 8, 1.0 / 16, 1.0 / 64, 1.0 / 384, -1.0 / 8};
    const Fat7Launch l = fat7_launch(ctx, fat7_fields(true, false));
    if (!l.work) return fail(ctx, LMB_ERR_CUDA, "out of device memory (smearing staples)");
    if ((rc = pack_links_to(ctx, thin, U, st))) return rc;
    if ((rc = fat7_planes(ctx, l, thin, lng, c_level1, st))) return rc;
    if ((rc = project_u3_planes(ctx, lng, w, st))) return rc;
    if ((rc = fat7_planes(ctx, l, w, fat, c_level2, st))) return rc;
    if ((rc = naik_planes(ctx, w, lng, st))) return rc;
    if ((rc = install_links(ctx, LMB_LINKS_FAT, st))) return rc;
    if ((rc = install_links(ctx, LMB_LINKS_LONG, st))) return rc;
    for (int mu = 0; mu < 4; mu++) {
      key.ptr[mu] = U[mu];
      key.epoch[mu] = epoch ? epoch[mu] : 0;
    }
    key.naik_epsilon = naik_epsilon;
    key.valid = epoch != nullptr;
  }
  if (X) {
    if ((rc = check_links_arg(ctx, (const void *const *)X, "fat link"))) return rc;
    if ((rc = unpack_links_from(ctx, X, ctx->links[LMB_LINKS_FAT].d, st))) return rc;
  }
  if (L) {
    if ((rc = check_links_arg(ctx, (const void *const *)L, "long link"))) return rc;
    if ((rc = unpack_links_from(ctx, L, ctx->links[LMB_LINKS_LONG].d, st))) return rc;
  }
  return LMB_OK;
}


int lmb_hisq_link_pullback(lmb_ctx *ctx, const void *const U[4], double naik_epsilon, double coefficient,
                           const void *result_cotangent, const void *psi, void *const dU[4], void *stream) {
  if (!ctx_ok(ctx)) return LMB_ERR_ARG;
  if (!ctx->geom_set) return fail(ctx, LMB_ERR_STATE, "lmb_set_geometry has not been called");
  int rc = check_links_arg(ctx, U, "thin link");
  if (rc) return rc;
  if ((rc = check_links_arg(ctx, (const void *const *)dU, "thin-link cotangent"))) return rc;
  if (!result_cotangent || !psi) return fail(ctx, LMB_ERR_ARG, "null fermion field");
  if (!std::isfinite(naik_epsilon) || !std::isfinite(coefficient))
    return fail(ctx, LMB_ERR_ARG, "naik_epsilon and coefficient must be finite");
  for (int mu = 0; mu < 4; mu++)
    for (int nu = 0; nu < 4; nu++)
      if (dU[mu] == U[nu]) return fail(ctx, LMB_ERR_ARG, "HISQ thin-link cotangents must not alias primal links");
  cudaStream_t st = as_stream(stream);
  const int64_t n = ctx->g.V;
  double2 *thin = (double2 *)workspace(ctx, "force_thin", sizeof(double2) * 36 * n);
  double2 *grad = (double2 *)workspace(ctx, "force_grad", sizeof(double2) * 36 * n);
  Field<PREC_DOUBLE, 3> dr, ps;
  if (!thin || !grad || !make_field(ctx, "force_dr", dr) || !make_field(ctx, "force_psi", ps))
    return fail(ctx, LMB_ERR_CUDA, "out of device memory (force)");
  if ((rc = pack_links_to(ctx, thin, U, st))) return rc;
  if ((rc = pack_in(ctx, dr, result_cotangent, st))) return rc;
  if ((rc = pack_in(ctx, ps, psi, st))) return rc;
  LMB_CUDA(ctx, cudaMemsetAsync(grad, 0, sizeof(double2) * 36 * n, st));
  if ((rc = hisq_pullback_planes(ctx, thin, dr, ps, naik_epsilon, coefficient, grad, st))) return rc;
  return accumulate_links_to(ctx, dU, grad, st);
}

int lmb_hisq_fermion_force(lmb_ctx *ctx, const void *const U[4], const uint64_t epoch[4], double mass,
                           double naik_epsilon, const void *phi, void *const dU[4], const lmb_cg_params *cg,
                           lmb_cg_result *result, void *stream) {
  if (!ctx_ok(ctx)) return LMB_ERR_ARG;
  if (!ctx->geom_set) return fail(ctx, LMB_ERR_STATE, "lmb_set_geometry has not been called");
  if (!cg || !result || !phi) return fail(ctx, LMB_ERR_ARG, "null argument");
  int rc = check_links_arg(ctx, U, "thin link");
  if (rc) return rc;
  if ((rc = check_links_arg(ctx, (const void *const *)dU, "force"))) return rc;
  cudaStream_t st = as_stream(stream);
  // the gradient's workspace, which the smearing then shares
  if (!fat7_launch(ctx, fat7_fields(true, true)).work)
    return fail(ctx, LMB_ERR_CUDA, "out of device memory (force staples)");
  // fat / long links for the solve (cached by thin-link pointer + epoch)
  if ((rc = lmb_hisq_links_from_thin(ctx, U, epoch, naik_epsilon, nullptr, nullptr, stream))) return rc;
  // eta = (D^+D)^-1 phi, chi = D eta, in padded scratch fields of the context geometry
  size_t padded = 3;
  for (int mu = 0; mu < 4; mu++) padded *= (size_t)ctx->pd.P[mu];
  const size_t elem = ctx->dtype == LMB_DTYPE_C128 ? 16 : 8;
  void *eta = workspace(ctx, "force_eta", padded * elem), *chi = workspace(ctx, "force_chi", padded * elem);
  if (!eta || !chi) return fail(ctx, LMB_ERR_CUDA, "out of device memory (force fields)");
  LMB_CUDA(ctx, cudaMemsetAsync(eta, 0, padded * elem, st));
  lmb_cg_params prm = *cg;
  prm.op = LMB_OP_HISQ;
  prm.mass = mass;
  prm.naik_epsilon = naik_epsilon;
  if ((rc = lmb_cg_ddagd(ctx, &prm, eta, phi, result, stream))) return rc;
  if ((rc = apply_dispatch(ctx, StaggeredPolicy{true, mass, naik_epsilon}, chi, eta, 0, PREC_DOUBLE, stream))) return rc;
  // dS/dU = -2 d/dU Re<chi, D(U) eta> with chi, eta fixed (dSFdU,
  // ext/LatticeMatricesEnzymeExt.jl:387-460)
  return lmb_hisq_link_pullback(ctx, U, naik_epsilon, -2.0, chi, eta, dU, stream);
}

int lmb_wilson_clover_link_pullback(lmb_ctx *ctx, const void *const U[4], double kappa, double csw,
                                    double coefficient, const void *result_cotangent, const void *psi,
                                    void *const dU[4], void *stream) {
  if (!ctx_ok(ctx)) return LMB_ERR_ARG;
  if (!ctx->geom_set) return fail(ctx, LMB_ERR_STATE, "lmb_set_geometry has not been called");
  int rc = check_links_arg(ctx, U, "primal link");
  if (rc) return rc;
  if ((rc = check_links_arg(ctx, (const void *const *)dU, "link cotangent"))) return rc;
  if (!result_cotangent || !psi) return fail(ctx, LMB_ERR_ARG, "null fermion field");
  if (!std::isfinite(kappa) || !std::isfinite(csw) || !std::isfinite(coefficient))
    return fail(ctx, LMB_ERR_ARG, "kappa, cSW and coefficient must be finite");
  for (int mu = 0; mu < 4; mu++)
    for (int nu = 0; nu < 4; nu++)
      if (dU[mu] == U[nu])
        return fail(ctx, LMB_ERR_ARG, "Wilson--clover link cotangents must not alias primal links");
  cudaStream_t st = as_stream(stream);
  const int64_t n = ctx->g.V;
  double2 *thin = (double2 *)workspace(ctx, "force_thin", sizeof(double2) * 36 * n);
  double2 *grad = (double2 *)workspace(ctx, "force_grad", sizeof(double2) * 36 * n);
  Field<PREC_DOUBLE, 12> dr, ps;
  if (!thin || !grad || !make_field(ctx, "force_dr12", dr) || !make_field(ctx, "force_psi12", ps))
    return fail(ctx, LMB_ERR_CUDA, "out of device memory (force)");
  if ((rc = pack_links_to(ctx, thin, U, st))) return rc;
  if ((rc = pack_in(ctx, dr, result_cotangent, st))) return rc;
  if ((rc = pack_in(ctx, ps, psi, st))) return rc;
  if ((rc = clover_pullback_planes(ctx, thin, dr, ps, kappa, csw, coefficient, grad, st))) return rc;
  return accumulate_links_to(ctx, dU, grad, st);
}

int lmb_wilson_clover_fermion_force(lmb_ctx *ctx, const void *const U[4], const uint64_t epoch[4], double kappa,
                                    double csw, const void *phi, void *const dU[4], const lmb_cg_params *cg,
                                    lmb_cg_result *result, void *stream) {
  if (!ctx_ok(ctx)) return LMB_ERR_ARG;
  if (!ctx->geom_set) return fail(ctx, LMB_ERR_STATE, "lmb_set_geometry has not been called");
  if (!cg || !result || !phi || !epoch) return fail(ctx, LMB_ERR_ARG, "null argument");
  int rc = check_links_arg(ctx, U, "primal link");
  if (rc) return rc;
  if ((rc = check_links_arg(ctx, (const void *const *)dU, "force"))) return rc;
  cudaStream_t st = as_stream(stream);
  if ((rc = lmb_links_upload(ctx, LMB_LINKS_THIN, U, epoch, stream))) return rc;
  // eta = (D^+D)^-1 phi, chi = D eta, in padded scratch fields of the context geometry
  size_t padded = 12;
  for (int mu = 0; mu < 4; mu++) padded *= (size_t)ctx->pd.P[mu];
  const size_t elem = ctx->dtype == LMB_DTYPE_C128 ? 16 : 8;
  void *eta = workspace(ctx, "force_eta12", padded * elem), *chi = workspace(ctx, "force_chi12", padded * elem);
  if (!eta || !chi) return fail(ctx, LMB_ERR_CUDA, "out of device memory (force fields)");
  LMB_CUDA(ctx, cudaMemsetAsync(eta, 0, padded * elem, st));
  lmb_cg_params prm = *cg;
  prm.op = csw != 0.0 ? LMB_OP_WILSON_CLOVER : LMB_OP_WILSON;
  prm.kappa = kappa;
  prm.csw = csw;
  if ((rc = lmb_cg_ddagd(ctx, &prm, eta, phi, result, stream))) return rc;
  if ((rc = apply_dispatch(ctx, WilsonPolicy{prm.op, kappa, csw}, chi, eta, 0, PREC_DOUBLE, stream))) return rc;
  // dS/dU = -2 d/dU Re<chi, D(U) eta> with chi, eta fixed
  return lmb_wilson_clover_link_pullback(ctx, U, kappa, csw, -2.0, chi, eta, dU, stream);
}


}  // extern "C"

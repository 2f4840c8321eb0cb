// lmb_clover_force.cuh -- hand-written adjoint of the Wilson-clover operator
// (FP64): gradient of f = coef Re<dr, D(U) psi> with respect to the links
// (wilson_clover_link_pullback!, WilsonCloverPullback.jl:342-403),
//   D psi = psi - kappa sum_mu [U_mu(x)(1 - g_mu)psi(x+mu) + U_mu(x-mu)^+(1 + g_mu)psi(x-mu)]
//           - kappa cSW sum_{mu<nu} G_mu_nu F_mu_nu psi,
//   F_mu_nu = (Q - Q^+)/8,  Q = the four plaquette leaves at x.
// Convention as lmb_hisq_force.cuh: df = Re sum conj(G_ij) dU_ij.
// Four stages, each gathering at the site it owns (no atomics):
//   1. hopping term: dU_mu(x) = c [dr(x) ((1-g)psi(x+mu))^+ + ((1+g)psi(x)) dr(x+mu)^+]
//      (WilsonDiracOperator.jl:382-411), fermion phases on wrapped hops;
//   2. cotangent of each F_mu_nu: dF(x) = c' sum_spin dr(x) (G psi(x))^+
//      (WilsonCloverPullback.jl:99-159), through F = (Q - Q^+)/8 the
//      anti-Hermitian H = (dF - dF^+)/8;
//   3. per plane (mu, nu), W_d(x) = H(x) U_d(x) + U_d(x) H(x+d) for d = mu, nu;
//   4. the links of the leaves.  U_mu(x) lies in two plaquettes of the plane,
//      and in each of them in the leaves anchored at its four corners, which
//      insert H there (WilsonCloverPullback.jl:161-292).  Gathering the two
//      insertions next to each of the other two sides into W_nu, and using
//      H^+ = -H, the eight leaves become four products
//        dU_mu(x) += W_nu(x) U_mu(x+nu) U_nu(x+mu)^+ - U_nu(x) U_mu(x+nu) W_nu(x+mu)^+
//                  + W_nu(y)^+ U_mu(y) U_nu(y+mu)    - U_nu(y)^+ U_mu(y) W_nu(y+mu)
//      with y = x - nu, and minus the same with mu and nu exchanged for
//      U_nu: 120 matrix products per site instead of some 500 with one
//      product chain per leaf and factor.
// 24^4: 4.67 -> 1.22 ms; 8^4: 0.41 -> 0.08 ms.  Stage 4 is bound as the Fat7
// stages are (lmb_fat7.cuh); two blocks of 254 registers, three spill.
#pragma once
#include "lmb_fat7.cuh"
#include "lmb_wilson.cuh"

namespace lmb {

// (1 + PM g_mu) psi as a full 12-component spinor (k = colour + 3 spin)
template <int PM, int MU>
LMB_D void spin_project_full(const Cx<double> *psi, Cx<double> *out) {
  Cx<double> h[6];
  project<PM, MU>(psi, h);
#pragma unroll
  for (int k = 0; k < 12; k++) out[k] = Cx<double>(0, 0);
  reconstruct<PM, MU>(out, h);
}

// G[a + 3b] += c sum_spin x[a + 3s] conj(y[b + 3s])
LMB_D void outer_spin_add(const Cx<double> *x, const Cx<double> *y, double c, Cx<double> *G) {
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) {
      Cx<double> v(0, 0);
#pragma unroll
      for (int s = 0; s < 4; s++) v = cfma_conj(y[b + 3 * s], x[a + 3 * s], v);
      G[a + 3 * b] = G[a + 3 * b] + c * v;
    }
}

template <int MU>
LMB_D void hop_outer(const Geom &g, int s, const int *c, const Field<PREC_DOUBLE, 12> &dr,
                     const Field<PREC_DOUBLE, 12> &psi, const Cx<double> *dr_x, const Cx<double> *psi_x,
                     double coef, double2 *dU) {
  int w;
  const int sp = fwd_site(g, s, c, MU, 1, &w);
  const bool ph = w && ((g.phase_mask >> MU) & 1);
  Cx<double> v[12], t[12], G[9];
  zero9(G);
  // U_mu(x) (1 - g) psi(x+mu) in (D psi)(x)
  psi.load(sp, t);
  if (ph) {
    const Cx<double> f(g.ph_fwd[MU][0], g.ph_fwd[MU][1]);
#pragma unroll
    for (int k = 0; k < 12; k++) t[k] = t[k] * f;
  }
  spin_project_full<-1, MU>(t, v);
  outer_spin_add(dr_x, v, coef, G);
  // U_mu(x)^+ (1 + g) psi(x) in (D psi)(x+mu), 1/phase when that hop wraps
  spin_project_full<+1, MU>(psi_x, v);
  if (ph) {
    const Cx<double> f(g.ph_bwd[MU][0], g.ph_bwd[MU][1]);
#pragma unroll
    for (int k = 0; k < 12; k++) v[k] = v[k] * f;
  }
  dr.load(sp, t);
  outer_spin_add(v, t, coef, G);
  store9(dU + (size_t)MU * 9 * g.V, g.V, s, G);
}

// stage 1: dU (36 planes, mu*9 + r + 3c) = coef * hopping-term gradient
template <int = 0>
__global__ void __launch_bounds__(128)
    wilson_outer_product_kernel(double2 *dU, const Field<PREC_DOUBLE, 12> dr, const Field<PREC_DOUBLE, 12> psi,
                                const Geom g, double coef) {
  const int s = blockIdx.x * 128 + threadIdx.x;
  if (s >= g.V) return;
  int c[4];
  site_coords(g, s, c);
  Cx<double> d[12], p[12];
  dr.load(s, d);
  psi.load(s, p);
  hop_outer<0>(g, s, c, dr, psi, d, p, coef, dU);
  hop_outer<1>(g, s, c, dr, psi, d, p, coef, dU);
  hop_outer<2>(g, s, c, dr, psi, d, p, coef, dU);
  hop_outer<3>(g, s, c, dr, psi, d, p, coef, dU);
}

// spin matrices of the clover term per plane (12, 13, 14, 23, 24, 34), as
// the block form of kernel_add_clover_term! (WilsonDiracCloverOperator.jl:
// 481-525): (G psi)_s for each colour
template <int PLANE>
LMB_D void clover_gamma_apply(const Cx<double> *p, Cx<double> *o) {
  const Cx<double> I(0, 1);
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const Cx<double> p1 = p[c], p2 = p[c + 3], p3 = p[c + 6], p4 = p[c + 9];
    Cx<double> o1, o2, o3, o4;
    if (PLANE == 0) {  // 12: diag(i, -i, i, -i)
      o1 = I * p1; o2 = -(I * p2); o3 = I * p3; o4 = -(I * p4);
    } else if (PLANE == 1) {  // 13
      o1 = -p2; o2 = p1; o3 = -p4; o4 = p3;
    } else if (PLANE == 2) {  // 14
      o1 = I * p2; o2 = I * p1; o3 = -(I * p4); o4 = -(I * p3);
    } else if (PLANE == 3) {  // 23
      o1 = I * p2; o2 = I * p1; o3 = I * p4; o4 = I * p3;
    } else if (PLANE == 4) {  // 24
      o1 = p2; o2 = -p1; o3 = -p4; o4 = p3;
    } else {  // 34: diag(i, -i, -i, i)
      o1 = I * p1; o2 = -(I * p2); o3 = -(I * p3); o4 = I * p4;
    }
    o[c] = o1;
    o[c + 3] = o2;
    o[c + 6] = o3;
    o[c + 9] = o4;
  }
}

// anti-Hermitian 3x3 matrices in five double2 planes: the imaginary diagonal
// (h0, h1), (h2, 0), then the entries (1,0), (2,0), (2,1)
constexpr int kAntiPlanes = 5;
LMB_D void load_anti(const double2 *F, int64_t V, int s, Cx<double> *h) {
  const double2 a = F[s], b = F[V + s], l10 = F[2 * V + s], l20 = F[3 * V + s], l21 = F[4 * V + s];
  h[0] = Cx<double>(0, a.x);
  h[4] = Cx<double>(0, a.y);
  h[8] = Cx<double>(0, b.x);
  h[1] = Cx<double>(l10.x, l10.y);
  h[2] = Cx<double>(l20.x, l20.y);
  h[5] = Cx<double>(l21.x, l21.y);
  h[3] = Cx<double>(-l10.x, l10.y);
  h[6] = Cx<double>(-l20.x, l20.y);
  h[7] = Cx<double>(-l21.x, l21.y);
}

template <int PLANE>
LMB_D void clover_cotangent_plane(const Cx<double> *d, const Cx<double> *p, double coef, double2 *H, int64_t V,
                                  int s) {
  Cx<double> gp[12], G[9];
  clover_gamma_apply<PLANE>(p, gp);
  zero9(G);
  outer_spin_add(d, gp, 0.125 * coef, G);
  double2 *o = H + (size_t)PLANE * kAntiPlanes * V;
  o[s] = make_double2(2 * G[0].im, 2 * G[4].im);
  o[V + s] = make_double2(2 * G[8].im, 0.0);
  o[2 * V + s] = make_double2(G[1].re - G[3].re, G[1].im + G[3].im);
  o[3 * V + s] = make_double2(G[2].re - G[6].re, G[2].im + G[6].im);
  o[4 * V + s] = make_double2(G[5].re - G[7].re, G[5].im + G[7].im);
}

// stage 2: H = (dF - dF^+)/8 of the six planes, dF = coef sum_spin dr (G psi)^+
template <int = 0>
__global__ void __launch_bounds__(128)
    clover_cotangent_kernel(double2 *H, const Field<PREC_DOUBLE, 12> dr, const Field<PREC_DOUBLE, 12> psi,
                            const Geom g, double coef) {
  const int s = blockIdx.x * 128 + threadIdx.x;
  if (s >= g.V) return;
  Cx<double> d[12], p[12];
  dr.load(s, d);
  psi.load(s, p);
  clover_cotangent_plane<0>(d, p, coef, H, g.V, s);
  clover_cotangent_plane<1>(d, p, coef, H, g.V, s);
  clover_cotangent_plane<2>(d, p, coef, H, g.V, s);
  clover_cotangent_plane<3>(d, p, coef, H, g.V, s);
  clover_cotangent_plane<4>(d, p, coef, H, g.V, s);
  clover_cotangent_plane<5>(d, p, coef, H, g.V, s);
}

// the two axes of a plane (12, 13, 14, 23, 24, 34), and the plane of two axes
LMB_HD int plane_first(int plane) { return plane < 3 ? 0 : plane < 5 ? 1 : 2; }
LMB_HD int plane_second(int plane) { return plane < 3 ? plane + 1 : plane < 5 ? plane - 1 : 3; }
LMB_HD int plane_of(int a, int b) {
  const int lo = a < b ? a : b, hi = a < b ? b : a;
  return lo == 0 ? hi - 1 : lo == 1 ? hi + 1 : 5;
}

// stage 3: W_d = H U_d + U_d H(x+d) of plane p0 + blockIdx.y / 2 for its first
// (blockIdx.y even) or second axis d, nine planes each
template <int = 0>
__global__ void __launch_bounds__(kFat7Threads)
    clover_insert_kernel(double2 *W, const double2 *U, const double2 *H, const Geom g, int p0) {
  const int s = blockIdx.x * kFat7Threads + threadIdx.x;
  if (s >= g.V) return;
  const int plane = p0 + blockIdx.y / 2, d = blockIdx.y & 1 ? plane_second(plane) : plane_first(plane);
  const double2 *Hp = H + (size_t)plane * kAntiPlanes * g.V;
  Cx<double> u[9], h[9], w[9], t[9];
  load9(U + (size_t)d * 9 * g.V, g.V, s, u);
  load_anti(Hp, g.V, s, h);
  mat3_mul(h, u, w);
  load_anti(Hp, g.V, s + step_up(g, s, d), h);
  mat3_mul(u, h, t);
#pragma unroll
  for (int k = 0; k < 9; k++) w[k] = w[k] + t[k];
  store9(W + (size_t)blockIdx.y * 9 * g.V, g.V, s, w);
}

// stage 4: dU_mu (mu = blockIdx.x mod 4) of the planes p0 .. p0 + np - 1
template <int = 0>
__global__ void __launch_bounds__(kFat7Threads, 2)
    clover_link_pullback_kernel(double2 *dU, const double2 *U, const double2 *W, const Geom g, const Fat7Tiles tl,
                                int p0, int np) {
  const int mu = blockIdx.x % 4;
  int s;
  if (!tile_site(g, tl.t[mu][0], blockIdx.x / 4, s)) return;
  const int64_t V = g.V;
  const double2 *Um = U + (size_t)mu * 9 * V;
  const int um = step_up(g, s, mu);
  Cx<double> acc[9];
  zero9(acc);
  bool any = false;
#pragma unroll 1
  for (int i = 0; i < 3; i++) {
    const int nu = axis_of(mu, i), plane = plane_of(mu, nu);
    if (plane < p0 || plane >= p0 + np) continue;
    any = true;
    const double2 *Un = U + (size_t)nu * 9 * V;
    const double2 *Wn = W + (size_t)(2 * (plane - p0) + (nu == plane_second(plane))) * 9 * V;
    const double sign = mu < nu ? 1.0 : -1.0;
    const int un = step_up(g, s, nu), dn = step_down(g, s, nu);
#pragma unroll 1
    for (int k = 0; k < 2; k++) {  // W on the near side, then (minus) on the far one
      const double2 *A = k ? Un : Wn, *B = k ? Wn : Un;
      const double f = k ? -sign : sign;
      Cx<double> m[9], b[9];
      load9(Um, V, s + un, m);
      load9(B, V, s + um, b);
#pragma unroll
      for (int e = 0; e < 9; e++) m[e] = f * m[e];
      tri_adj(acc, A, V, s, m, b);
      load9(Um, V, s + dn, m);
      load9(B, V, s + dn + um, b);
#pragma unroll
      for (int e = 0; e < 9; e++) m[e] = f * m[e];
      tri_fwd(acc, A, V, s + dn, m, b);
    }
  }
  if (!any) return;
  double2 *o = dU + (size_t)mu * 9 * V;
  axpy9(acc, 1.0, o, V, s);
  store9(o, V, s, acc);
}

}  // namespace lmb

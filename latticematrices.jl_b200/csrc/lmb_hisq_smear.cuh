// lmb_hisq_smear.cuh -- 3x3 link algebra, U(3) projection and Naik links of the
// HISQ smearing (FP64).
//
// Fat7 (+ Lepage) lives in lmb_fat7.cuh.  U(3) projection W = V (V^+V)^{-1/2}
// with the trigonometric eigenvalues and Cayley-Hamilton coefficients
// (HISQFullSmearing.jl:1-77); Naik links L_mu(x) = W_mu(x) W_mu(x+mu) W_mu(x+2mu)
// (HISQFullSmearing.jl:136-195).
//
// Link planes: (mu*9 + r + 3c) * V + s (double2), as the link caches.
// Single-direction fields (staples): (r + 3c) * V + s.
#pragma once
#include "lmb_pack.cuh"

namespace lmb {

constexpr int kSmearThreads = 128;

LMB_D void load9(const double2 *F, int64_t V, int s, Cx<double> *m) {
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const double2 t = F[k * V + s];
    m[k] = Cx<double>(t.x, t.y);
  }
}
LMB_D void store9(double2 *F, int64_t V, int s, const Cx<double> *m) {
#pragma unroll
  for (int k = 0; k < 9; k++) F[k * V + s] = make_double2(m[k].re, m[k].im);
}
// c = a * b^+
LMB_D void mat3_mul_adj(const Cx<double> *a, const Cx<double> *b, Cx<double> *c) {
  Cx<double> t[9];
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int col = 0; col < 3; col++) {
      Cx<double> v = a[r] * conj(b[col]);
      v = cfma_conj(b[col + 3], a[r + 3], v);
      v = cfma_conj(b[col + 6], a[r + 6], v);
      t[r + 3 * col] = v;
    }
#pragma unroll
  for (int k = 0; k < 9; k++) c[k] = t[k];
}
// c = a^+ * b
LMB_D void mat3_adj_mul(const Cx<double> *a, const Cx<double> *b, Cx<double> *c) {
  Cx<double> t[9];
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int col = 0; col < 3; col++) {
      Cx<double> v = conj(a[3 * r]) * b[3 * col];
      v = cfma_conj(a[3 * r + 1], b[1 + 3 * col], v);
      v = cfma_conj(a[3 * r + 2], b[2 + 3 * col], v);
      t[r + 3 * col] = v;
    }
#pragma unroll
  for (int k = 0; k < 9; k++) c[k] = t[k];
}

LMB_D int nb_site(const Geom &g, int s, int mu, int d) {
  int c[4], w;
  site_coords(g, s, c);
  return d > 0 ? fwd_site(g, s, c, mu, d, &w) : bwd_site(g, s, c, mu, -d, &w);
}

// (V^+V)^{-1/2} for the U(3) projection (HISQFullSmearing.jl:1-77):
// Q = V^+V, its eigenvalues g0, g1, g2 from the trigonometric solution of
// the characteristic cubic (coefficients from traces of Q, Q^2, Q^3), each
// floored at the machine epsilon, and Q^{-1/2} = f0 + f1 Q + f2 Q^2 by
// Cayley-Hamilton, f_k symmetric functions of sqrt(g_i).  Returns Q, Q^2,
// Q^{-1/2} and the elementary symmetric functions u, v, w of the sqrt(g_i)
// (the U(3) pullback needs them).  The smearing and the force share it, so
// both use the same branch thresholds.
struct U3Inverse {
  Cx<double> Q[9], Q2[9], inv[9];
  double u, v, w;
};
LMB_D void u3_inverse_sqrt(const Cx<double> *Vm, U3Inverse &r) {
  mat3_adj_mul(Vm, Vm, r.Q);
  mat3_mul(r.Q, r.Q, r.Q2);
  double c0 = 0, trQ2 = 0, trQ3 = 0;
  for (int i = 0; i < 3; i++) {
    c0 += r.Q[i + 3 * i].re;
    trQ2 += r.Q2[i + 3 * i].re;
    for (int j = 0; j < 3; j++) trQ3 += (r.Q2[i + 3 * j] * r.Q[j + 3 * i]).re;
  }
  const double c1 = trQ2 / 2, c2 = trQ3 / 3;
  double S = c1 / 3 - c0 * c0 / 18;
  double g0, g1, g2;
  if (fabs(S) < 1e-7) {
    g0 = g1 = g2 = c0 / 3;
  } else {
    S = sqrt(fmax(S, 0.0));
    const double R = c2 / 2 - c0 * c1 / 3 + c0 * c0 * c0 / 27;
    double ratio = R / (S * S * S);
    ratio = fmin(1.0, fmax(-1.0, ratio));
    const double theta = acos(ratio);
    const double tpt = 2.0943951023931954923;  // 2 pi / 3
    const double center = c0 / 3, amp = 2 * S;
    g0 = center + amp * cos(theta / 3 - tpt);
    g1 = center + amp * cos(theta / 3);
    g2 = center + amp * cos(theta / 3 + tpt);
  }
  const double fl = 2.220446049250313e-16;
  g0 = fmax(g0, fl);
  g1 = fmax(g1, fl);
  g2 = fmax(g2, fl);
  const double u = sqrt(g0) + sqrt(g1) + sqrt(g2);
  const double v = sqrt(g0 * g1) + sqrt(g0 * g2) + sqrt(g1 * g2);
  const double w = sqrt(g0 * g1 * g2);
  const double den = w * (u * v - w);
  const double f0 = (-w * (u * u + v) + u * v * v) / den;
  const double f1 = (-w - u * u * u + 2 * u * v) / den;
  const double f2 = u / den;
#pragma unroll
  for (int k = 0; k < 9; k++) r.inv[k] = f1 * r.Q[k] + f2 * r.Q2[k];
  for (int i = 0; i < 3; i++) r.inv[i + 3 * i] = r.inv[i + 3 * i] + Cx<double>(f0, 0);
  r.u = u;
  r.v = v;
  r.w = w;
}

// W = V (V^+V)^{-1/2}
LMB_D void u3_project(const Cx<double> *Vm, Cx<double> *W) {
  U3Inverse r;
  u3_inverse_sqrt(Vm, r);
  mat3_mul(Vm, r.inv, W);
}

template <int = 0>
__global__ void __launch_bounds__(kSmearThreads)
    u3_project_kernel(double2 *W, const double2 *Vall, int64_t n) {
  const int64_t t = (int64_t)blockIdx.x * kSmearThreads + threadIdx.x;
  if (t >= 4 * n) return;
  const int mu = (int)(t / n);
  const int s = (int)(t - (int64_t)mu * n);
  Cx<double> v[9], w[9];
  load9(Vall + (size_t)mu * 9 * n, n, s, v);
  u3_project(v, w);
  store9(W + (size_t)mu * 9 * n, n, s, w);
}

// L_mu(x) = W_mu(x) W_mu(x+mu) W_mu(x+2mu)
template <int = 0>
__global__ void __launch_bounds__(kSmearThreads)
    naik_kernel(double2 *Lall, const double2 *W, const Geom g) {
  const int64_t t = (int64_t)blockIdx.x * kSmearThreads + threadIdx.x;
  if (t >= 4 * g.V) return;
  const int mu = (int)(t / g.V);
  const int s = (int)(t - (int64_t)mu * g.V);
  const double2 *Wm = W + (size_t)mu * 9 * g.V;
  const int s1 = nb_site(g, s, mu, 1), s2 = nb_site(g, s1, mu, 1);
  Cx<double> a[9], b[9];
  load9(Wm, g.V, s, a);
  load9(Wm, g.V, s1, b);
  mat3_mul(a, b, a);
  load9(Wm, g.V, s2, b);
  mat3_mul(a, b, a);
  store9(Lall + (size_t)mu * 9 * g.V, g.V, s, a);
}

// unpack 36 link planes to four padded (3,3,...) fields
template <typename TOUT>
__global__ void __launch_bounds__(256)
    unpack_links_kernel(TOUT *U0, TOUT *U1, TOUT *U2, TOUT *U3, const double2 *src, const Geom g,
                        const Padded pd) {
  const int s = blockIdx.x * 256 + threadIdx.x;
  if (s >= g.V) return;
  int c[4];
  site_coords(g, s, c);
  const int64_t ps = padded_site(pd, c) * 9;
  TOUT *U[4] = {U0, U1, U2, U3};
#pragma unroll
  for (int mu = 0; mu < 4; mu++) {
    if (!U[mu]) continue;
#pragma unroll
    for (int k = 0; k < 9; k++) {
      const double2 t = src[(mu * 9 + k) * g.V + s];
      U[mu][ps + k].x = t.x;
      U[mu][ps + k].y = t.y;
    }
  }
}

}  // namespace lmb

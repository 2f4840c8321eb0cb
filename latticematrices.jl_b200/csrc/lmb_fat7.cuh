// lmb_fat7.cuh -- Fat7 (+ Lepage) smearing and its adjoint in four stages.
//
// For a link direction mu with transverse axes (a, b, c) and the transport
//   T_n(M)(x) = T+_n(M) + T-_n(M),
//   T+_n(M)(x) = U_n(x) M(x+n) U_n(x+mu)^+,
//   T-_n(M)(x) = U_n(x-n)^+ M(x-n) U_n(x-n+mu),
// the factorised Fat7 of a field X (X = U_mu in the smearing) is
//   S_n  = T_n(X)                                              (stage 1)
//   M_n  = c3 X + c5 sum_{k != n} S_k + c7 [T_a(S_c) + T_c(S_a)]  (stage 2)
//   M+-_n = M_n + cL T+-_n(X)
//   F(X) = c1 X + sum_n [T+_n(M+_n) + T-_n(M-_n)]               (stage 3)
// ({a, c} the axes other than n): the three-, five- and seven-link staples of
// HISQSmearing.jl:768-974 with the outermost transport of every path taken
// once on the sum of its arguments.  The Lepage paths (n,n,mu,-n,-n) and
// (-n,-n,mu,n,n) are T+_n(T+_n(X)) + T-_n(T-_n(X)) and ride on that transport.
//
// Adjoint: T+_n and T-_n are each other's adjoints in M, so F is its own
// adjoint in X.  With G = dV_mu, S, P+- from X = U_mu (c3 = 0) and R, N+- from
// X = G, the cotangents are dU_mu += F(G) and, for each axis nu, with
//   Q(A, B)(z) = A(z) U_nu(z+mu) B(z+nu)^+ + A(z-mu)^+ U_nu(z-mu) B(z-mu+nu),
//   dU_nu += Q(G, P+) + Q(P-, G) + Q(N-, U_mu) + Q(U_mu, N+)
//            + c7 [Q(R_a, S_c) + Q(S_c, R_a) + Q(R_c, S_a) + Q(S_a, R_c)]  (stage 4)
// ({a, c} the axes other than nu).  Smearing levels are recomputed, not
// stored, and every kernel gathers to the site it owns (no atomics).
//
// What bounds it: every product gathers two or three matrices of 144 B per
// site through L1 and L2 (the stages move 11 to 15 TB/s there, and 3 to 4 TB/s
// of DRAM), then FP64 arithmetic (108 DFMA per product, the pipe 25 to 37 %
// busy).  A launch per transport wrote and re-read every intermediate field;
// the fused stages move 25 matrix fields of DRAM traffic per direction instead
// of 50, and their four-dimensional blocks of sites find about a third of
// the neighbours in L1.  24^3 x 48 smearing: 10.3 -> 7.1 ms (the chain of
// launches took 6.9 ms for the two Fat7 levels and 1.3 ms for Lepage paths
// evaluated link by link); 24^4 link gradient: 22.0 -> 12.2 ms; at 8^4, where
// launches count (some 130 of them became 8), 2.64 -> 0.35 ms.  Occupancy is
// 3 blocks of 168 registers; 2 and 4 blocks measured the same for the
// staples.
#pragma once
#include "lmb_hisq_smear.cuh"

namespace lmb {

constexpr int kFat7Threads = 128;

// block of sites t[0] x t[1] x t[2] x t[3] (at most kFat7Threads), n[d] of
// them along d
struct SiteTile {
  int t[4], n[4];
};

// one block shape for each direction mu and slot (transverse axis) of a launch
struct Fat7Tiles {
  SiteTile t[4][3];
};

LMB_D bool tile_site(const Geom &g, const SiteTile &tl, unsigned tile, int &s) {
  int b = (int)tile, l = (int)threadIdx.x;
  bool in = l < tl.t[0] * tl.t[1] * tl.t[2] * tl.t[3];
  s = 0;
#pragma unroll
  for (int d = 0; d < 4; d++) {
    const int qb = b / tl.n[d], ql = l / tl.t[d];
    const int x = (b - qb * tl.n[d]) * tl.t[d] + (l - ql * tl.t[d]);
    in = in && x < g.L[d];
    s += x * g.stride[d];
    b = qb;
    l = ql;
  }
  return in && b == 0;
}

// index offset of the neighbour of site s at +1 / -1 along d
LMB_D int step_up(const Geom &g, int s, int d) {
  const int x = (s / g.stride[d]) % g.L[d];
  return x == g.L[d] - 1 ? (1 - g.L[d]) * g.stride[d] : g.stride[d];
}
LMB_D int step_down(const Geom &g, int s, int d) {
  const int x = (s / g.stride[d]) % g.L[d];
  return x == 0 ? (g.L[d] - 1) * g.stride[d] : -g.stride[d];
}

// acc += A(s) m b^+ with A streamed by rows from memory
LMB_D void tri_adj(Cx<double> *acc, const double2 *A, int64_t V, int s, const Cx<double> *m, const Cx<double> *b) {
#pragma unroll
  for (int r = 0; r < 3; r++) {
    Cx<double> a[3], t[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const double2 v = A[(r + 3 * j) * V + s];
      a[j] = Cx<double>(v.x, v.y);
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      t[c] = a[0] * m[3 * c];
      t[c] = cfma(a[1], m[3 * c + 1], t[c]);
      t[c] = cfma(a[2], m[3 * c + 2], t[c]);
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
#pragma unroll
      for (int k = 0; k < 3; k++) acc[r + 3 * c] = cfma_conj(b[c + 3 * k], t[k], acc[r + 3 * c]);
    }
  }
}
// acc += A(s)^+ m b
LMB_D void tri_fwd(Cx<double> *acc, const double2 *A, int64_t V, int s, const Cx<double> *m, const Cx<double> *b) {
#pragma unroll
  for (int r = 0; r < 3; r++) {
    Cx<double> a[3], t[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const double2 v = A[(j + 3 * r) * V + s];
      a[j] = Cx<double>(v.x, v.y);
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      t[c] = conj(a[0]) * m[3 * c];
      t[c] = cfma_conj(a[1], m[3 * c + 1], t[c]);
      t[c] = cfma_conj(a[2], m[3 * c + 2], t[c]);
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
#pragma unroll
      for (int k = 0; k < 3; k++) acc[r + 3 * c] = cfma(t[k], b[k + 3 * c], acc[r + 3 * c]);
    }
  }
}

LMB_D void zero9(Cx<double> *a) {
#pragma unroll
  for (int k = 0; k < 9; k++) a[k] = Cx<double>(0, 0);
}
// acc += c * F(s)
LMB_D void axpy9(Cx<double> *acc, double c, const double2 *F, int64_t V, int s) {
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const double2 t = F[k * V + s];
    acc[k].re += c * t.x;
    acc[k].im += c * t.y;
  }
}

// acc += T+_n(M)(s) / T-_n(M)(s); Un the links of direction n, um = step up
// along mu from s (down: from s - n, the same coordinate)
LMB_D void transport_up(Cx<double> *acc, const double2 *M, const double2 *Un, int64_t V, int s, int un, int um) {
  Cx<double> m[9], b[9];
  load9(M, V, s + un, m);
  load9(Un, V, s + um, b);
  tri_adj(acc, Un, V, s, m, b);
}
LMB_D void transport_down(Cx<double> *acc, const double2 *M, const double2 *Un, int64_t V, int s, int dn, int um) {
  Cx<double> m[9], b[9];
  load9(M, V, s + dn, m);
  load9(Un, V, s + dn + um, b);
  tri_fwd(acc, Un, V, s + dn, m, b);
}

LMB_D int axis_of(int mu, int slot) { return slot < mu ? slot : slot + 1; }

// One application of the Fat7 map: X (9 planes per direction at stride 9 V)
// and its intermediates, three 9-plane fields each, per direction handled in
// this launch at stride `per_mu`.  Mm = Mp where there is no Lepage term (the
// two arguments agree then); with it Mp holds T+(X) between stages 1 and 2.
struct Fat7Field {
  const double2 *X;
  double2 *S, *Mp, *Mm;
  double c3;
};

// stage 1: S_n = T_n(X) (LEPAGE: and T+_n(X) in Mp_n)
template <int NF, bool LEPAGE>
__global__ void __launch_bounds__(kFat7Threads, 3)
    fat7_three_kernel(const Geom g, const Fat7Tiles tl, const double2 *U, const Fat7Field f0, const Fat7Field f1,
                      int mu0, int64_t per_mu) {
  const int slot = blockIdx.x % 3, mu = mu0 + blockIdx.y;
  int s;
  if (!tile_site(g, tl.t[blockIdx.y][slot], blockIdx.x / 3, s)) return;
  const int64_t V = g.V;
  const int n = axis_of(mu, slot);
  const double2 *Un = U + (size_t)n * 9 * V;
  const int un = step_up(g, s, n), dn = step_down(g, s, n), um = step_up(g, s, mu);
#pragma unroll 1
  for (int i = 0; i < NF; i++) {
    const Fat7Field &f = i ? f1 : f0;
    const double2 *X = f.X + (size_t)mu * 9 * V;
    const size_t at = (size_t)blockIdx.y * per_mu + (size_t)slot * 9 * V;
    Cx<double> acc[9];
    zero9(acc);
    transport_up(acc, X, Un, V, s, un, um);
    if (LEPAGE) store9(f.Mp + at, V, s, acc);
    transport_down(acc, X, Un, V, s, dn, um);
    store9(f.S + at, V, s, acc);
  }
}

// stage 2: M_n (LEPAGE: M+_n over T+_n(X), and M-_n)
template <int NF, bool LEPAGE>
__global__ void __launch_bounds__(kFat7Threads, 3)
    fat7_five_kernel(const Geom g, const Fat7Tiles tl, const double2 *U, const Fat7Field f0, const Fat7Field f1,
                     int mu0, int64_t per_mu, double c5, double c7, double cL) {
  const int slot = blockIdx.x % 3, mu = mu0 + blockIdx.y;
  int s;
  if (!tile_site(g, tl.t[blockIdx.y][slot], blockIdx.x / 3, s)) return;
  const int64_t V = g.V;
  const int um = step_up(g, s, mu);
  const int other[2] = {slot == 0 ? 1 : 0, slot == 2 ? 1 : 2};
#pragma unroll 1
  for (int i = 0; i < NF; i++) {
    const Fat7Field &f = i ? f1 : f0;
    double2 *S = f.S + (size_t)blockIdx.y * per_mu;
    const size_t at = (size_t)blockIdx.y * per_mu + (size_t)slot * 9 * V;
    Cx<double> acc[9];
    zero9(acc);
#pragma unroll 1
    for (int k = 0; k < 2; k++) {
      const int ka = other[0], kc = other[1];
      const int a = axis_of(mu, k ? kc : ka);
      const double2 *Ua = U + (size_t)a * 9 * V, *Sc = S + (size_t)(k ? ka : kc) * 9 * V;
      transport_up(acc, Sc, Ua, V, s, step_up(g, s, a), um);
      transport_down(acc, Sc, Ua, V, s, step_down(g, s, a), um);
    }
#pragma unroll
    for (int k = 0; k < 9; k++) acc[k] = c7 * acc[k];
    axpy9(acc, c5, S + (size_t)other[0] * 9 * V, V, s);
    axpy9(acc, c5, S + (size_t)other[1] * 9 * V, V, s);
    if (f.c3 != 0.0) axpy9(acc, f.c3, f.X + (size_t)mu * 9 * V, V, s);
    if (LEPAGE) {
      Cx<double> p[9], q[9];
      load9(f.Mp + at, V, s, p);
      load9(S + (size_t)slot * 9 * V, V, s, q);
#pragma unroll
      for (int k = 0; k < 9; k++) {
        q[k] = acc[k] + cL * (q[k] - p[k]);
        p[k] = acc[k] + cL * p[k];
      }
      store9(f.Mp + at, V, s, p);
      store9(f.Mm + at, V, s, q);
    } else {
      store9(f.Mp + at, V, s, acc);
    }
  }
}

// stage 3: out_mu (+)= c1 X + sum_n T+_n(M+_n) + T-_n(M-_n)
template <bool ACCUMULATE>
__global__ void __launch_bounds__(kFat7Threads, 3)
    fat7_sum_kernel(const Geom g, const Fat7Tiles tl, const double2 *U, double2 *out, const Fat7Field f, int mu0,
                    int64_t per_mu, double c1) {
  const int mu = mu0 + blockIdx.y;
  int s;
  if (!tile_site(g, tl.t[blockIdx.y][0], blockIdx.x, s)) return;
  const int64_t V = g.V;
  const int um = step_up(g, s, mu);
  Cx<double> acc[9];
  zero9(acc);
#pragma unroll 1
  for (int slot = 0; slot < 3; slot++) {
    const int n = axis_of(mu, slot);
    const size_t at = (size_t)blockIdx.y * per_mu + (size_t)slot * 9 * V;
    const double2 *Un = U + (size_t)n * 9 * V;
    transport_up(acc, f.Mp + at, Un, V, s, step_up(g, s, n), um);
    transport_down(acc, f.Mm + at, Un, V, s, step_down(g, s, n), um);
  }
  axpy9(acc, c1, f.X + (size_t)mu * 9 * V, V, s);
  double2 *o = out + (size_t)mu * 9 * V;
  if (ACCUMULATE) axpy9(acc, 1.0, o, V, s);
  store9(o, V, s, acc);
}

// acc += Q(A, B)(z): up = U_nu(z+mu) with A, B at z, z+nu, and down =
// U_nu(z-mu) with A, B at z-mu, z-mu+nu
LMB_D void grad_pair(Cx<double> *acc, const double2 *A, const double2 *B, const Cx<double> *up,
                     const Cx<double> *down, int64_t V, int z, int un, int dm) {
  Cx<double> b[9];
  load9(B, V, z + un, b);
  tri_adj(acc, A, V, z, up, b);
  load9(B, V, z + dm + un, b);
  tri_fwd(acc, A, V, z + dm, down, b);
}

// Two blocks of 255 registers hold both U_nu across the eight pairs (a third
// of the gathers); three blocks that loaded them per pair measured 4 % slower.
// stage 4: dU_nu of the directions mu0 .. mu0 + nmu - 1 (fu: X = U, fg: X = G)
template <int = 0>
__global__ void __launch_bounds__(kFat7Threads, 2)
    fat7_grad_kernel(const Geom g, const Fat7Tiles tl, const double2 *U, double2 *dU, const Fat7Field fu,
                     const Fat7Field fg, int mu0, int nmu, int64_t per_mu, double c7) {
  const int nu = blockIdx.x % 4;
  if (nmu == 1 && nu == mu0) return;
  int z;
  if (!tile_site(g, tl.t[0][0], blockIdx.x / 4, z)) return;
  const int64_t V = g.V;
  const double2 *Un = U + (size_t)nu * 9 * V;
  const int un = step_up(g, z, nu);
  double2 *o = dU + (size_t)nu * 9 * V;
#pragma unroll 1
  for (int i = 0; i < nmu; i++) {
    const int mu = mu0 + i;
    if (mu == nu) continue;
    const int um = step_up(g, z, mu), dm = step_down(g, z, mu);
    const int slot = nu < mu ? nu : nu - 1;
    const size_t base = (size_t)i * per_mu;
    const size_t n = base + (size_t)slot * 9 * V;
    const size_t a = base + (size_t)(slot == 0 ? 1 : 0) * 9 * V, c = base + (size_t)(slot == 2 ? 1 : 2) * 9 * V;
    const double2 *X = fu.X + (size_t)mu * 9 * V, *G = fg.X + (size_t)mu * 9 * V;
    Cx<double> acc[9], up[9], down[9];
    zero9(acc);
    load9(Un, V, z + um, up);
    load9(Un, V, z + dm, down);
#pragma unroll 1
    for (int k = 0; k < 8; k++) {
      if (k == 4) {  // the first four carry c7
#pragma unroll
        for (int e = 0; e < 9; e++) acc[e] = c7 * acc[e];
      }
      const double2 *A, *B;
      if (k < 4) {
        const double2 *r = fg.S + (k & 1 ? c : a), *q = fu.S + (k & 1 ? a : c);
        A = k & 2 ? q : r;
        B = k & 2 ? r : q;
      } else {
        A = k == 4 ? G : k == 5 ? fu.Mm + n : k == 6 ? fg.Mm + n : X;
        B = k == 4 ? fu.Mp + n : k == 5 ? G : k == 6 ? X : fg.Mp + n;
      }
      grad_pair(acc, A, B, up, down, V, z, un, dm);
    }
    axpy9(acc, 1.0, o, V, z);
    store9(o, V, z, acc);
  }
}

}  // namespace lmb

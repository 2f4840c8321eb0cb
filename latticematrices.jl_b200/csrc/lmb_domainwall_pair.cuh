// lmb_domainwall_pair.cuh -- one-pass domain-wall stencils on pairs of
// fifth-coordinate neighbours (FP32 and int16 storage, even L5).
//
// A thread owns the slices s and s + 1 (s even) of one 4D point: lane x and
// lane y of packed FP32 (lmb_pair.cuh).  The two sites are adjacent in memory
// (the fifth coordinate is the fastest), so one 256-bit load serves both, and
// they share their eight links, which are loaded, decoded and completed to
// three rows once for two sites.  Of the neighbours in s that F takes, half
// are the other lane: lane y's s - 1 is lane x and lane x's s + 1 is lane y,
// so D5 reads 1.5 spinors per site and hop (its own, half a spinor below and
// above the pair) instead of two, and D5^+ exchanges half of Z through shared
// memory instead of all of it.
//
// No unit stands at its limit: at 16^3x32x12 on int16 fields a D5 (a D5^+) issues
// in 51 (49) % of the slots, the FMA pipe is 46 (45) % busy, L1 44 (36) %, and it
// moves 0.8 (1.5) TB/s of DRAM and 6 (7) through L2, at 16 warps per SM; its
// packed arithmetic alone takes about 85 us.  At that size a D5 takes 195 us on int16 fields (one site per thread: 242)
// and a D5^+ with the CG update 178 (231); the solves take 217 ms on int16
// (265) and 262 ms on FP32 fields (290).  The other way round, int16 on three
// blocks of 168 registers and FP32 on four of 128, they take 223 and 284 ms;
// with the link in both lanes of 36 registers 223 and 269 ms on three blocks.
// FP32 links of 18 reals for int16 fields, which spare the decode and the third
// row, measured slower (241 ms).
#pragma once
#include "lmb_domainwall.cuh"
#include "lmb_pair_hop.cuh"

namespace lmb {

LMB_D float2 dw_lanes(const double *v, int s0, int s1, double f0, double f1) {
  return f2((float)(f0 * v[s0]), (float)(f1 * v[s1]));
}

// (lo.x from q, lo.y from lane x of p) and (hi.x from lane y of p, hi.y from q)
LMB_D Cx2 dw_below(const Cx<float> &q, const Cx2 &p) { return Cx2(f2(q.re, p.re.x), f2(q.im, p.im.x)); }
LMB_D Cx2 dw_above(const Cx2 &p, const Cx<float> &q) { return Cx2(f2(p.re.y, q.re), f2(p.im.y, q.im)); }

// resident blocks per SM: int16 words leave room for four (128 registers, D5
// spills 170 bytes), FP32 ones for three
template <class SF> struct DWPairBlocks { static constexpr int value = 3; };
template <> struct DWPairBlocks<Field<PREC_HALF, 12>> { static constexpr int value = 4; };

// slices and coefficients of a pair: i0 = index of slice s within the point,
// below / above the slices next to the pair, and for D5 the factors of
// Y = b psi + c F psi
struct DWPair {
  int s, below, above;
  float2 b, cl, ch;
};

// projected half spinor of Y at the point y4 (D5)
template <int PM, int MU, class SF>
LMB_D void dw_Y_proj2(const SF &psi, int64_t base, const DWPair &d, Cx2 *h) {
  Cx2 p[12];
  load_adj(psi, base + d.s, p);
  project<PM, MU>(p, h);
#pragma unroll
  for (int k = 0; k < 6; k++) h[k] = Cx2(d.b * h[k].re, d.b * h[k].im);
  Cx<float> q[12];
  load_part<0, 6>(psi, base + d.below, q);
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const Cx2 v = dw_below(q[k], p[k]);
    h[k] = Cx2(fma2(d.cl, v.re, h[k].re), fma2(d.cl, v.im, h[k].im));
  }
  load_part<6, 12>(psi, base + d.above, q);
  Cx2 u[12], t[6];
#pragma unroll
  for (int k = 6; k < 12; k++) u[k] = dw_above(p[k], q[k]);
  project_lower<PM, MU>(u, t);
#pragma unroll
  for (int k = 0; k < 6; k++) h[k] = Cx2(fma2(d.ch, t[k].re, h[k].re), fma2(d.ch, t[k].im, h[k].im));
}

// one link for both lanes, U h and U^+ h: an entry is put into both lanes where
// it is used, for the two colour vectors at once, so that the link takes 18
// registers and not 36
LMB_D void shared_mul_half(const Cx<float> *u, const Cx2 *h, Cx2 *o) {
#pragma unroll
  for (int r = 0; r < 3; r++) {
    const Cx2 e(f2(u[r].re), f2(u[r].im));
    o[r] = e * h[0];
    o[r + 3] = e * h[3];
  }
#pragma unroll
  for (int k = 1; k < 3; k++)
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const Cx2 e(f2(u[r + 3 * k].re), f2(u[r + 3 * k].im));
      o[r] = cfma(e, h[k], o[r]);
      o[r + 3] = cfma(e, h[k + 3], o[r + 3]);
    }
}
LMB_D void shared_adj_mul_half(const Cx<float> *u, const Cx2 *h, Cx2 *o) {
#pragma unroll
  for (int r = 0; r < 3; r++) {
    const Cx2 e(f2(u[3 * r].re), f2(-u[3 * r].im));
    o[r] = e * h[0];
    o[r + 3] = e * h[3];
  }
#pragma unroll
  for (int k = 1; k < 3; k++)
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const Cx2 e(f2(u[3 * r + k].re), f2(u[3 * r + k].im));
      o[r] = cfma_conj(e, h[k], o[r]);
      o[r + 3] = cfma_conj(e, h[k + 3], o[r + 3]);
    }
}

template <int DAG, int MU, bool FUSED, class SF, class G>
LMB_D void dw_hop2(const Geom &g, int x4, const int *c, int L5, const DWPair &d, const SF &in, const G &U,
                   Cx2 *acc) {
  constexpr int FPM = DAG ? +1 : -1;
  constexpr int BPM = -FPM;
  Cx2 h[6], uh[6];
  Cx<float> us[9];
  int wrap;
  {
    const int sp = fwd_site(g, x4, c, MU, 1, &wrap);
    if constexpr (FUSED) {
      dw_Y_proj2<FPM, MU>(in, (int64_t)sp * L5, d, h);
    } else {
      load_project_adj<FPM, MU>(in, (int64_t)sp * L5 + d.s, h);
    }
    if (wrap && ((g.phase_mask >> MU) & 1)) phase2(h, g.ph_fwd[MU], 1, 1);
    U.load(MU, x4, us);
    shared_mul_half(us, h, uh);
    reconstruct<FPM, MU>(acc, uh);
  }
  {
    const int sm = bwd_site(g, x4, c, MU, 1, &wrap);
    if constexpr (FUSED) {
      dw_Y_proj2<BPM, MU>(in, (int64_t)sm * L5, d, h);
    } else {
      load_project_adj<BPM, MU>(in, (int64_t)sm * L5 + d.s, h);
    }
    if (wrap && ((g.phase_mask >> MU) & 1)) phase2(h, g.ph_bwd[MU], 1, 1);
    U.load(MU, sm, us);
    shared_adj_mul_half(us, h, uh);
    reconstruct<BPM, MU>(acc, uh);
  }
}

template <int DAG, bool FUSED, class SF, class G>
LMB_D void dw_hops2(const Geom &g, int x4, int L5, const DWPair &d, const SF &in, const G &U, Cx2 *acc) {
  int c[4];
  site_coords(g, x4, c);
#pragma unroll
  for (int k = 0; k < 12; k++) acc[k] = cx2_zero();
  dw_hop2<DAG, 0, FUSED>(g, x4, c, L5, d, in, U, acc);
  dw_hop2<DAG, 1, FUSED>(g, x4, c, L5, d, in, U, acc);
  dw_hop2<DAG, 2, FUSED>(g, x4, c, L5, d, in, U, acc);
  dw_hop2<DAG, 3, FUSED>(g, x4, c, L5, d, in, U, acc);
}

LMB_D DWPair dw_pair(int s, int L5) {
  DWPair d;
  d.s = s;
  d.below = s == 0 ? L5 - 1 : s - 1;
  d.above = s + 2 == L5 ? 0 : s + 2;
  return d;
}

// D5: one thread per pair of slices
template <class SF, class G, class Epi>
__global__ void __launch_bounds__(kDslashThreads, DWPairBlocks<SF>::value)
    dw_forward_pair_kernel(const Geom g, const SF psi, const G U, const DWParams dw, Epi epi) {
  if (epi.skip()) return;
  const int L5 = dw.L5, half = L5 / 2;
  const int64_t j = (int64_t)blockIdx.x * kDslashThreads + threadIdx.x;
  const bool active = j < g.V * half;
  Cx2 out[12];
  if (active) {
    const int x4 = (int)(j / half);
    DWPair d = dw_pair(2 * (int)(j - (int64_t)x4 * half), L5);
    const float flo = d.s == 0 ? (float)-dw.mass : 1.f, fhi = d.s + 2 == L5 ? (float)-dw.mass : 1.f;
    const float2 c = dw_lanes(dw.c, d.s, d.s + 1, 1.0, 1.0);
    d.b = dw_lanes(dw.b, d.s, d.s + 1, 1.0, 1.0);
    d.cl = c * f2(flo, 1.f);
    d.ch = c * f2(1.f, fhi);
    Cx2 acc[12];
    dw_hops2<0, true>(g, x4, L5, d, psi, U, acc);
    const int64_t base = (int64_t)x4 * L5;
    Cx2 p[12];
    Cx<float> q[12];
    load_adj(psi, base + d.s, p);
    load_part<0, 6>(psi, base + d.below, q);
    load_part<6, 12>(psi, base + d.above, q);
    const float2 a = dw_lanes(dw.a, d.s, d.s + 1, 1.0, 1.0), diag = f2((float)(4.0 + dw.M));
    const float2 mh = f2(-0.5f);
#pragma unroll
    for (int k = 0; k < 12; k++) {
      const Cx2 f = k < 6 ? dw_below(q[k], p[k]) : dw_above(p[k], q[k]);
      const float2 ff = k < 6 ? f2(flo, 1.f) : f2(1.f, fhi);
      const Cx2 fk(ff * f.re, ff * f.im);
      const Cx2 y(fma2(c, fk.re, d.b * p[k].re), fma2(c, fk.im, d.b * p[k].im));
      const float2 re = fma2(diag, y.re, fma2(mh, acc[k].re, p[k].re - fk.re));
      const float2 im = fma2(diag, y.im, fma2(mh, acc[k].im, p[k].im - fk.im));
      out[k] = Cx2(a * re, a * im);
    }
  }
  epi.pair_adj((int)(active ? 2 * j : 0), active, out);
}

// D5^+: blocks of `npts` whole 4D points (npts * L5 / 2 <= kDslashThreads)
template <class SF, class G, class Epi>
__global__ void __launch_bounds__(kDslashThreads, DWPairBlocks<SF>::value)
    dw_adjoint_pair_kernel(const Geom g, const SF psi, const G U, const DWParams dw, int npts, Epi epi) {
  // of every pair, what its neighbours take: spins 1, 2 of lane x (the pair
  // below it) and spins 3, 4 of lane y (the pair above)
  __shared__ float zs[24 * kDslashThreads];
  if (epi.skip()) return;
  const int L5 = dw.L5, half = L5 / 2;
  const int t = threadIdx.x;
  const int gx = t / half, j = t - gx * half;
  const int64_t x4 = (int64_t)blockIdx.x * npts + gx;
  const bool active = gx < npts && x4 < g.V;
  const DWPair d = dw_pair(2 * j, L5);
  const int64_t base = x4 * L5;
  Cx2 z[12];
  if (active) {
    Cx2 p[12];
    dw_hops2<1, false>(g, (int)x4, L5, d, psi, U, z);
    load_adj(psi, base + d.s, p);
    const float2 a = dw_lanes(dw.a, d.s, d.s + 1, 1.0, 1.0), diag = f2((float)(4.0 + dw.M)), mh = f2(-0.5f);
#pragma unroll
    for (int k = 0; k < 12; k++) {
      z[k] = Cx2(a * fma2(diag, p[k].re, mh * z[k].re), a * fma2(diag, p[k].im, mh * z[k].im));
      zs[(2 * k) * kDslashThreads + t] = k < 6 ? z[k].re.x : z[k].re.y;
      zs[(2 * k + 1) * kDslashThreads + t] = k < 6 ? z[k].im.x : z[k].im.y;
    }
  }
  __syncthreads();
  Cx2 out[12];
  if (active) {
    const double flo = d.s + 2 == L5 ? -dw.mass : 1.0, fhi = d.s == 0 ? -dw.mass : 1.0;
    const float2 zl = dw_lanes(dw.c, d.s + 1, d.above, 1.0, flo), zh = dw_lanes(dw.c, d.below, d.s, fhi, 1.0);
    const float2 pl = dw_lanes(dw.a, d.s + 1, d.above, -1.0, -flo), ph = dw_lanes(dw.a, d.below, d.s, -fhi, -1.0);
    const float2 a = dw_lanes(dw.a, d.s, d.s + 1, 1.0, 1.0), b = dw_lanes(dw.b, d.s, d.s + 1, 1.0, 1.0);
    const int up = gx * half + (d.above >> 1), dn = gx * half + (d.below >> 1);
    Cx2 p[12];
    Cx<float> q[12];
    load_adj(psi, base + d.s, p);
    load_part<0, 6>(psi, base + d.above, q);
    load_part<6, 12>(psi, base + d.below, q);
#pragma unroll
    for (int k = 0; k < 12; k++) {
      const int o = k < 6 ? up : dn;
      const Cx<float> zq(zs[(2 * k) * kDslashThreads + o], zs[(2 * k + 1) * kDslashThreads + o]);
      const Cx2 f = k < 6 ? dw_above(p[k], q[k]) : dw_below(q[k], p[k]);
      const Cx2 zn = k < 6 ? dw_above(z[k], zq) : dw_below(zq, z[k]);
      const float2 pf = k < 6 ? pl : ph, zf = k < 6 ? zl : zh;
      out[k] = Cx2(fma2(zf, zn.re, fma2(b, z[k].re, fma2(pf, f.re, a * p[k].re))),
                   fma2(zf, zn.im, fma2(b, z[k].im, fma2(pf, f.im, a * p[k].im))));
    }
  }
  epi.pair_adj((int)(active ? base + d.s : 0), active, out);
}

}  // namespace lmb

// lmb_evenodd_pair.cuh -- even/odd hops on pairs of checkerboard neighbours
// (int16 storage, x extent a multiple of 4).
//
// A thread owns the checkerboard indices cb, cb + 1 (cb even) of one parity:
// two sites of the same row, two apart in x, as the lanes of packed FP32.  The
// y, z and t neighbours sit at the same place of their row, so they are such a
// pair again and one 256-bit load per plane serves both lanes, as it does for
// the links and clover blocks of the two sites.  Along x one of the two hops
// stays at the same index (a pair), the other moves by one; which one depends
// on the row's parity, and both load lane by lane.
//
// The one-site kernel decodes, projects and multiplies one site per thread in
// scalar FP32.  24^3x48 clover, int16: two hops with K1 109 -> 90 us, with K2 118
// -> 100 us, the solve 40.2 -> 35.3 ms (two blocks per SM 38.3, four 39.1).  No
// unit stands at its limit: a hop (40 to 52 us) moves 3.3 to 3.5 TB/s of DRAM and 7
// to 8 through L2, issues in 35 to 41 % of the slots, the FMA pipe is 39 to 45 %
// busy, at 12 warps per SM in 168 registers.
#pragma once
#include "lmb_evenodd.cuh"
#include "lmb_pair_hop.cuh"

namespace lmb {

// hops of direction MU into the sites s, s + 2 (s = the site of cb, x extent
// L0, coordinates c); es = parity-ordered index of s
template <int DAG, int MU, class SF, class G>
LMB_D void eo_hop2(const Geom &g, int s, int64_t es, int p, const int *c, const SF &in, const G &U, Cx2 *acc) {
  constexpr int FPM = DAG ? +1 : -1;
  constexpr int BPM = -FPM;
  const bool ph = (g.phase_mask >> MU) & 1;
  const int64_t other = (int64_t)(1 - p) * (g.V / 2);
  Cx2 h[6], uh[6], u[9];
  int w0, w1;
  {
    const int n0 = fwd_site(g, s, c, MU, 1, &w0);
    if constexpr (MU == 0) {
      w1 = c[0] + 3 >= g.L[0];  // w0 is 0: x + 1 stays in the row unless s + 2 ends it
      const int n1 = w1 ? n0 + 2 - g.L[0] : n0 + 2;
      load_project2<FPM, MU>(in, n0 >> 1, n1 >> 1, h);
    } else {
      w1 = w0;
      load_project_adj<FPM, MU>(in, n0 >> 1, h);
    }
    if (ph && (w0 | w1)) phase2(h, g.ph_fwd[MU], w0, w1);
    load_adj(U, MU, es, u);
    su3_mul_half(u, h, uh);
    reconstruct<FPM, MU>(acc, uh);
  }
  {
    const int n0 = bwd_site(g, s, c, MU, 1, &w0);
    if constexpr (MU == 0) {
      w1 = 0;
      const int n1 = s + 1;
      load_project2<BPM, MU>(in, n0 >> 1, n1 >> 1, h);
      if (ph && w0) phase2(h, g.ph_bwd[MU], w0, w1);
      load2(U, MU, other + (n0 >> 1), other + (n1 >> 1), u);
    } else {
      w1 = w0;
      load_project_adj<BPM, MU>(in, n0 >> 1, h);
      if (ph && w0) phase2(h, g.ph_bwd[MU], w0, w1);
      load_adj(U, MU, other + (n0 >> 1), u);
    }
    su3_adj_mul_half(u, h, uh);
    reconstruct<BPM, MU>(acc, uh);
  }
}

template <class C>
LMB_D void clover_apply2(const C &A, int64_t s, Cx2 *v) {
#pragma unroll
  for (int blk = 0; blk < 2; blk++) {
    float2 a[36];
    Cx2 o[6];
    load_adj(A, blk, s, a);
    herm6_mul(a, v + 6 * blk, o);
#pragma unroll
    for (int k = 0; k < 6; k++) v[6 * blk + k] = o[k];
  }
}

// as eo_hop_kernel, two checkerboard sites per thread
template <int DAG, int WMODE, bool AINV, bool CL, class SF, class G, class C, class Epi>
__global__ void __launch_bounds__(kDslashThreads, 3)
    eo_hop_pair_kernel(const Geom g, const int p, const SF in, const SF W, const G U, const C A, const C Ainv,
                       const float c1, const float c2, Epi epi) {
  if (epi.skip()) return;
  const int64_t cb = 2 * ((int64_t)blockIdx.x * kDslashThreads + threadIdx.x);
  const bool active = cb < g.V / 2;
  Cx2 v[12];
  if (active) {
    int c[4];
    const int s = cb_site(g, (int)cb, p, c);
    const int64_t es = (int64_t)p * (g.V / 2) + cb;
#pragma unroll
    for (int k = 0; k < 12; k++) v[k] = cx2_zero();
    eo_hop2<DAG, 0>(g, s, es, p, c, in, U, v);
    eo_hop2<DAG, 1>(g, s, es, p, c, in, U, v);
    eo_hop2<DAG, 2>(g, s, es, p, c, in, U, v);
    eo_hop2<DAG, 3>(g, s, es, p, c, in, U, v);
#pragma unroll
    for (int k = 0; k < 12; k++) v[k] = Cx2(f2(c2) * v[k].re, f2(c2) * v[k].im);
    if constexpr (WMODE != 0) {
      Cx2 w[12];
      load_adj(W, cb, w);
      if constexpr (WMODE == 2 && CL) clover_apply2(A, es, w);
#pragma unroll
      for (int k = 0; k < 12; k++) v[k] = Cx2(fma2(f2(c1), w[k].re, v[k].re), fma2(f2(c1), w[k].im, v[k].im));
    }
    if constexpr (AINV && CL) clover_apply2(Ainv, es, v);
  }
  epi.pair_adj((int)(active ? cb : 0), active, v);
}

}  // namespace lmb

// lmb_pair_hop.cuh -- projected half spinors, links and clover blocks of two
// sites in packed FP32 for FP32 and int16 storage: what the domain-wall and
// even/odd pair stencils share beyond lmb_pair.cuh.
#pragma once
#include "lmb_pair.cuh"
#include "lmb_wilson.cuh"

namespace lmb {

LMB_D void ld256f(const float4 *p, float4 &a, float4 &b) {
  int4 ia, ib;
  ld256(reinterpret_cast<const int4 *>(p), ia, ib);
  a = as_f4(ia);
  b = as_f4(ib);
}

// adjacent pairs of FP32 spinors, reconstruct-12 links and clover blocks
LMB_D void load_adj(const Field<PREC_SINGLE, 12> &f, int64_t s, Cx2 *v) {
#pragma unroll
  for (int k = 0; k < 6; k++) {
    float4 a, b;
    ld256f(f.data + k * f.V + s, a, b);
    v[2 * k] = Cx2(f2(a.x, b.x), f2(a.y, b.y));
    v[2 * k + 1] = Cx2(f2(a.z, b.z), f2(a.w, b.w));
  }
}
LMB_D void load_adj(const Gauge12<PREC_SINGLE> &U, int mu, int64_t s, Cx2 *u) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    float4 a, b;
    ld256f(U.data + (mu * 3 + k) * U.V + s, a, b);
    const int e0 = 2 * k, e1 = 2 * k + 1;
    u[(e0 / 3) + 3 * (e0 % 3)] = Cx2(f2(a.x, b.x), f2(a.y, b.y));
    u[(e1 / 3) + 3 * (e1 % 3)] = Cx2(f2(a.z, b.z), f2(a.w, b.w));
  }
  su3_third_row(u);
}
LMB_D void load_adj(const Clover<PREC_SINGLE> &A, int blk, int64_t s, float2 *v) {
#pragma unroll
  for (int k = 0; k < 9; k++) {
    float4 a, b;
    ld256f(A.data + (blk * 9 + k) * A.V + s, a, b);
    v[4 * k] = f2(a.x, b.x);
    v[4 * k + 1] = f2(a.y, b.y);
    v[4 * k + 2] = f2(a.z, b.z);
    v[4 * k + 3] = f2(a.w, b.w);
  }
}

// projected half spinors of the sites s, s + 1 (s even) and of two sites;
// int16 words are projected before their offset is taken off (project_raw)
template <int PM, int MU>
LMB_D void load_project_adj(const Field<PREC_SINGLE, 12> &f, int64_t s, Cx2 *h) {
  Cx2 p[12];
  load_adj(f, s, p);
  project<PM, MU>(p, h);
}
template <int PM, int MU>
LMB_D void load_project_adj(const Field<PREC_HALF, 12> &f, int64_t s, Cx2 *h) {
  Cx2 p[12];
  float2 nc2;
  load_adj_raw(f, s, p, nc2);
  project_raw<PM, MU>(p, nc2, h);
}
template <int PM, int MU>
LMB_D void load_project2(const Field<PREC_SINGLE, 12> &f, int64_t s0, int64_t s1, Cx2 *h) {
  Cx2 p[12];
  load2(f, s0, s1, p);
  project<PM, MU>(p, h);
}
template <int PM, int MU>
LMB_D void load_project2(const Field<PREC_HALF, 12> &f, int64_t s0, int64_t s1, Cx2 *h) {
  Cx2 p[12];
  float2 nc2;
  load2_raw(f, s0, s1, p, nc2);
  project_raw<PM, MU>(p, nc2, h);
}

}  // namespace lmb

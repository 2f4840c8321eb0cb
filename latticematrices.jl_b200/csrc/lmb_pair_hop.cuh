// lmb_pair_hop.cuh -- projected half spinors of two sites in packed FP32: what
// the pair stencils of the domain wall (FP32 and int16 storage) and of the
// even/odd solve (int16) take beyond lmb_pair.cuh.
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

// an adjacent pair of FP32 spinors
LMB_D void load_adj(const Field<PREC_SINGLE, 12> &f, int64_t s, Cx2 *v) {
#pragma unroll
  for (int k = 0; k < 6; k++) {
    float4 a, b;
    ld256f(f.data + k * f.V + s, a, b);
    v[2 * k] = Cx2(f2(a.x, b.x), f2(a.y, b.y));
    v[2 * k + 1] = Cx2(f2(a.z, b.z), f2(a.w, b.w));
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
LMB_D void load_project2(const Field<PREC_HALF, 12> &f, int64_t s0, int64_t s1, Cx2 *h) {
  Cx2 p[12];
  float2 nc2;
  load2_raw(f, s0, s1, p, nc2);
  project_raw<PM, MU>(p, nc2, h);
}

}  // namespace lmb

// lmb_small.cuh -- conjugate gradient on small lattices: all iterations of a
// solve (up to the next FP64 reliable update) in one cooperative launch.
//
// On a lattice of a few thousand sites the three kernels of an iteration
// (lmb_solver.cuh) take their launches and their longest thread, not their
// bytes: at 8^4 in FP64 K1 is 32 blocks of threads that each walk eight hops
// one after the other (11.5 us), K2 the same (13.5 us), with a two-stage
// reduction at the end of both.  Here a block of eight warps owns tiles of 32
// sites and each warp takes one of the eight hops of those sites, so a site's
// hops run side by side on all SMs; the partial results meet in shared memory,
// where four warps (one per spin) finish the site and its vector update.  The
// phases of an iteration
//   A  tmp = D p, <tmp, tmp>    B  x += alpha p, r -= alpha D^+ tmp, <r, r>
//   C  p = r + beta p
// are separated by grid barriers, which carry the partial sums of A and B; all
// blocks take the same scalar step from the same total.  (Forming r + beta p
// at the neighbours instead of C and its barrier gained 3 % at 8^4 and lost 8 %
// from 12^4 on.)  The links and clover blocks of a block's tiles stay in
// its L1 from one iteration to the next.
//
// Fields that other blocks write during the launch are read through L2
// (ld.global.cg): neither the read-only path nor L1 is coherent within a
// kernel.  Every barrier wait is bounded: a block that gives up returns, and the
// others, which then wait in vain for it, do the same; the caller sees that the
// iteration count did not advance.
#pragma once
#include "lmb_solver.cuh"

namespace lmb {

constexpr int kSmallThreads = 256;   // eight warps: (direction, sense)
constexpr int kSmallTile = 32;       // sites per tile, one per lane
// resident blocks per SM: FP64 hops need 128 registers, the FP32 ones fit 80
template <int PS>
constexpr int small_min_blocks() { return PS == PREC_DOUBLE ? 2 : 3; }

// ---------------------------------------------------------------------------
// storage: whole sites, and the three components of one group, through L2
// ---------------------------------------------------------------------------
template <int NC>
LMB_D void cg_load(const Field<PREC_DOUBLE, NC> &f, int64_t s, Cx<double> *v) {
#pragma unroll
  for (int k = 0; k < NC; k++) {
    const double2 t = __ldcg(f.data + k * f.V + s);
    v[k] = Cx<double>(t.x, t.y);
  }
}
LMB_D void cg_load(const Field<PREC_SINGLE, 12> &f, int64_t s, Cx<float> *v) {
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const float4 t = __ldcg(f.data + k * f.V + s);
    v[2 * k] = Cx<float>(t.x, t.y);
    v[2 * k + 1] = Cx<float>(t.z, t.w);
  }
}
LMB_D void cg_load(const Field<PREC_SINGLE, 3> &f, int64_t s, Cx<float> *v) {
  const float4 a = __ldcg(f.data + s);
  const float2 b = __ldcg(f.last() + s);
  v[0] = Cx<float>(a.x, a.y);
  v[1] = Cx<float>(a.z, a.w);
  v[2] = Cx<float>(b.x, b.y);
}
template <int NC>
LMB_D void cg_load(const Field<PREC_HALF, NC> &f, int64_t s, Cx<float> *v) {
  const Dec16 d = dec16_of_base(__ldcg(f.norm + s));
#pragma unroll
  for (int k = 0; k < Field<PREC_HALF, NC>::kPlanes; k++) {
    const int4 t = __ldcg(f.data + k * f.V + s);
    const int w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (4 * k + j < NC) {
        const float2 q = dec_pair(w[j], d);
        v[4 * k + j] = Cx<float>(q.x, q.y);
      }
  }
}

// components K0 .. K1 - 1 of a site (the planes that hold them)
template <int K0, int K1>
LMB_D void cg_part(const Field<PREC_DOUBLE, 12> &f, int64_t i, Cx<double> *v) {
#pragma unroll
  for (int k = K0; k < K1; k++) {
    const double2 t = __ldcg(f.data + k * f.V + i);
    v[k] = Cx<double>(t.x, t.y);
  }
}
template <int K0, int K1>
LMB_D void cg_part(const Field<PREC_SINGLE, 12> &f, int64_t i, Cx<float> *v) {
#pragma unroll
  for (int p = K0 / 2; p < K1 / 2; p++) {
    const float4 t = __ldcg(f.data + p * f.V + i);
    v[2 * p] = Cx<float>(t.x, t.y);
    v[2 * p + 1] = Cx<float>(t.z, t.w);
  }
}
template <int K0, int K1>
LMB_D void cg_part(const Field<PREC_HALF, 12> &f, int64_t i, Cx<float> *v) {
  const Dec16 d = dec16_of_base(__ldcg(f.norm + i));
#pragma unroll
  for (int p = K0 / 4; p < (K1 + 3) / 4; p++) {
    const int4 t = __ldcg(f.data + p * f.V + i);
    const int w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (4 * p + j >= K0 && 4 * p + j < K1) {
        const float2 q = dec_pair(w[j], d);
        v[4 * p + j] = Cx<float>(q.x, q.y);
      }
  }
}

// address of component k of a site
template <int NC>
LMB_D double2 *comp_at(const Field<PREC_DOUBLE, NC> &f, int64_t s, int k) { return f.data + k * f.V + s; }
LMB_D float2 *comp_at(const Field<PREC_SINGLE, 12> &f, int64_t s, int k) {
  return reinterpret_cast<float2 *>(f.data + (k >> 1) * f.V + s) + (k & 1);
}
LMB_D float2 *comp_at(const Field<PREC_SINGLE, 3> &f, int64_t s, int k) {
  return k < 2 ? reinterpret_cast<float2 *>(f.data + s) + k : f.last() + s;
}
template <int NC>
LMB_D int *comp_at(const Field<PREC_HALF, NC> &f, int64_t s, int k) {
  return reinterpret_cast<int *>(f.data + (k >> 2) * f.V + s) + (k & 3);
}

// the components 3 q .. 3 q + 2 of the thread's own site
template <int PS, int NC, typename R>
LMB_D void own_load(const Field<PS, NC> &f, int64_t s, int q, Cx<R> *v) {
  Dec16 d;
  if constexpr (PS == PREC_HALF) d = dec16_of_base(__ldcg(f.norm + s));
#pragma unroll
  for (int k = 0; k < 3; k++) {
    if constexpr (PS == PREC_HALF) {
      const float2 t = dec_pair(__ldcg(comp_at(f, s, 3 * q + k)), d);
      v[k] = Cx<R>(t.x, t.y);
    } else {
      const auto t = __ldcg(comp_at(f, s, 3 * q + k));
      v[k] = Cx<R>(t.x, t.y);
    }
  }
}
// int16 storage scales a whole site: the groups exchange their largest
// magnitudes in `mag` (all threads of the block call this)
template <int PS, int NC, typename R>
LMB_D void own_store(const Field<PS, NC> &f, int64_t s, int q, bool mine, const Cx<R> *v, float (*mag)[kSmallTile]) {
  constexpr int G = NC / 3;
  if constexpr (PS == PREC_HALF) {
    const int lane = threadIdx.x & 31;
    float m = 0.f;
    if (mine) {
#pragma unroll
      for (int k = 0; k < 3; k++) m = fmaxf(m, fmaxf(fabsf((float)v[k].re), fabsf((float)v[k].im)));
      mag[q][lane] = m;
    }
    if constexpr (G > 1) __syncthreads();
    if (mine) {
#pragma unroll
      for (int i = 0; i < G; i++) m = fmaxf(m, mag[i][lane]);
      const int e = enc_exponent(m);
      const float inv = enc_inv(e);
#pragma unroll
      for (int k = 0; k < 3; k++)
        *comp_at(f, s, 3 * q + k) =
            enc_word(fmaf((float)v[k].re, inv, 8421376.0f), fmaf((float)v[k].im, inv, 8421376.0f));
      if (q == 0) f.norm[s] = enc_base(e);
      if (NC == 3) *comp_at(f, s, 3) = (int)0x80008000u;  // q = 0
    }
  } else if (mine) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      if constexpr (PS == PREC_DOUBLE) *comp_at(f, s, 3 * q + k) = make_double2(v[k].re, v[k].im);
      else *comp_at(f, s, 3 * q + k) = make_float2((float)v[k].re, (float)v[k].im);
    }
  }
}

// an application reads its field through this
template <int PS, int NC>
struct SrcField {
  Field<PS, NC> f;
  typedef typename Real<PS>::type R;
  LMB_D void load(int64_t i, Cx<R> *v) const { cg_load(f, i, v); }
  template <int K0, int K1>
  LMB_D void part(int64_t i, Cx<R> *v) const { cg_part<K0, K1>(f, i, v); }
  LMB_D void own(int64_t i, int q, Cx<R> *v) const { own_load(f, i, q, v); }
};

// ---------------------------------------------------------------------------
// operators: sites() of them (one lane of a tile each), phases(DAG) passes per
// application, each ending in finish<DAG, PH>; every pass but the last stores
// to `mid`, which the next one reads; kWaves, the tiles per resident block up to
// which the one launch is the faster way (lmb_small_host.cuh).  One hop of a site, and one group's components of D psi from the
// eight hops in shared memory (element i of warp w's hop at hops[w][i][lane])
// ---------------------------------------------------------------------------
template <typename R>
struct SmallHops {
  R v[8][12][kSmallTile];
};

template <typename R>
LMB_D void put_hop(SmallHops<R> &sm, int w, int n, const Cx<R> *h) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 6; k++)
    if (k < n) {
      sm.v[w][2 * k][lane] = h[k].re;
      sm.v[w][2 * k + 1][lane] = h[k].im;
    }
}
template <typename R>
LMB_D Cx<R> get_hop(const SmallHops<R> &sm, int w, int k) {
  const int lane = threadIdx.x & 31;
  return Cx<R>(sm.v[w][2 * k][lane], sm.v[w][2 * k + 1][lane]);
}

// rows 3 HI .. 3 HI + 2 of a Hermitian 6x6 (herm6_mul) times v
template <int HI, typename R>
LMB_D void herm6_rows(const R *a, const Cx<R> *v, Cx<R> *o) {
#pragma unroll
  for (int r = 0; r < 3; r++) {
    const int i = 3 * HI + r;
    o[r] = a[i] * v[i];
#pragma unroll
    for (int j = 0; j < 6; j++) {
      if (j == i) continue;
      const int hi = i > j ? i : j, lo = i > j ? j : i, k = 6 + hi * (hi - 1) + 2 * lo;
      const Cx<R> e(a[k], a[k + 1]);
      o[r] = i > j ? cfma(e, v[j], o[r]) : cfma_conj(e, v[j], o[r]);
    }
  }
}

// spin Q of the reconstructed hop of warp W (reconstruct<PM, MU>), and of all
// eight
template <int DAG, int Q, int W, typename R>
LMB_D void add_spin(const SmallHops<R> &sm, Cx<R> *acc) {
  constexpr int MU = W >> 1;
  constexpr bool P = (W & 1) ? DAG == 0 : DAG == 1;  // PM > 0
  constexpr int half = Q < 2 ? Q : ((MU < 2) ? 3 - Q : Q - 2);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const Cx<R> h = get_hop(sm, W, k + 3 * half);
    if constexpr (Q < 2) {
      acc[k] = acc[k] + h;
    } else if constexpr (MU == 0 || MU == 2) {
      constexpr bool plus = (MU == 2 && Q == 3) ? !P : P;
      acc[k] = plus ? acc[k] + mul_i(h) : acc[k] - mul_i(h);
    } else {
      constexpr bool plus = (MU == 1 && Q == 2) ? P : !P;
      acc[k] = plus ? acc[k] + h : acc[k] - h;
    }
  }
}
template <int DAG, int Q, typename R>
LMB_D void sum_spin(const SmallHops<R> &sm, Cx<R> *acc) {
#pragma unroll
  for (int k = 0; k < 3; k++) acc[k] = Cx<R>(0, 0);
  add_spin<DAG, Q, 0>(sm, acc);
  add_spin<DAG, Q, 1>(sm, acc);
  add_spin<DAG, Q, 2>(sm, acc);
  add_spin<DAG, Q, 3>(sm, acc);
  add_spin<DAG, Q, 4>(sm, acc);
  add_spin<DAG, Q, 5>(sm, acc);
  add_spin<DAG, Q, 6>(sm, acc);
  add_spin<DAG, Q, 7>(sm, acc);
}

template <int PS, class G, class CL, bool CLOVER>
struct SmallWilson {
  static constexpr int NC = 12;
  typedef typename Real<PS>::type R;
  G U;
  CL A;
  R kappa;
  Field<PS, 12> mid;  // unused: one pass
  static constexpr int kWaves = PS == PREC_SINGLE ? 5 : PS == PREC_DOUBLE ? (CLOVER ? 3 : 4) : (CLOVER ? 1 : 2);
  static constexpr int phases(int) { return 1; }
  LMB_HD int64_t sites(const Geom &g) const { return g.V; }

  template <int DAG, int W, class Src>
  LMB_D void hop_w(const Geom &g, int s, const int *c, const Src &in, SmallHops<R> &sm) const {
    constexpr int MU = W >> 1, BACK = W & 1;
    constexpr int PM = (DAG ? +1 : -1) * (BACK ? -1 : +1);
    int wrap;
    const int n = BACK ? bwd_site(g, s, c, MU, 1, &wrap) : fwd_site(g, s, c, MU, 1, &wrap);
    Cx<R> p[12], h[6], uh[6], u[9];
    in.load(n, p);
    U.load(MU, BACK ? n : s, u);
    project<PM, MU>(p, h);
    if (wrap && ((g.phase_mask >> MU) & 1)) scale_phase(h, 6, BACK ? g.ph_bwd[MU] : g.ph_fwd[MU]);
    if (BACK) su3_adj_mul_half(u, h, uh);
    else su3_mul_half(u, h, uh);
    put_hop(sm, W, 6, uh);
  }
  template <int DAG, int PH, class Src>
  LMB_D void hop(int w, const Geom &g, int s, const Src &in, SmallHops<R> &sm) const {
    int c[4];
    site_coords(g, s, c);
    switch (w) {
      case 0: hop_w<DAG, 0>(g, s, c, in, sm); break;
      case 1: hop_w<DAG, 1>(g, s, c, in, sm); break;
      case 2: hop_w<DAG, 2>(g, s, c, in, sm); break;
      case 3: hop_w<DAG, 3>(g, s, c, in, sm); break;
      case 4: hop_w<DAG, 4>(g, s, c, in, sm); break;
      case 5: hop_w<DAG, 5>(g, s, c, in, sm); break;
      case 6: hop_w<DAG, 6>(g, s, c, in, sm); break;
      default: hop_w<DAG, 7>(g, s, c, in, sm); break;
    }
  }
  template <int DAG, int Q, class Src>
  LMB_D void spin(int s, const Src &in, const SmallHops<R> &sm, Cx<R> *out) const {
    Cx<R> acc[3];
    sum_spin<DAG, Q>(sm, acc);
    if constexpr (CLOVER) {
      R a[36];
      Cx<R> v[6], o[3];
      A.load(Q >> 1, s, a);
      in.own(s, Q & 2, v);
      in.own(s, (Q & 2) + 1, v + 3);
      herm6_rows<(Q & 1)>(a, v, o);
#pragma unroll
      for (int k = 0; k < 3; k++) out[k] = o[k] - kappa * acc[k];
    } else {
      Cx<R> v[3];
      in.own(s, Q, v);
#pragma unroll
      for (int k = 0; k < 3; k++) out[k] = v[k] - kappa * acc[k];
    }
  }
  template <int DAG, int PH, class Src>
  LMB_D void finish(int q, const Geom &, int s, const Src &in, const SmallHops<R> &sm, Cx<R> *out) const {
    switch (q) {
      case 0: spin<DAG, 0>(s, in, sm, out); break;
      case 1: spin<DAG, 1>(s, in, sm, out); break;
      case 2: spin<DAG, 2>(s, in, sm, out); break;
      default: spin<DAG, 3>(s, in, sm, out); break;
    }
  }
};

// staggered (NAIK = false) and HISQ: a warp's hop is its fat and its Naik link
template <int PS, class GF, class GL, bool NAIK>
struct SmallStaggered {
  static constexpr int NC = 3;
  typedef typename Real<PS>::type R;
  GF X;
  GL L;
  R mass, fc, lc;  // of D; D^+ negates fc and lc
  Field<PS, 3> mid;  // unused: one pass
  static constexpr int kWaves = NAIK ? (PS == PREC_HALF ? 2 : 3) : (PS == PREC_DOUBLE ? 4 : 5);
  static constexpr int phases(int) { return 1; }
  LMB_HD int64_t sites(const Geom &g) const { return g.V; }

  template <int MU, int BACK, int D, class G, class Src>
  LMB_D void link_hop(const Geom &g, int s, const int *c, const Src &in, const G &U, R f, Cx<R> *acc) const {
    int w;
    const int n = shift_site_any(g, s, c, MU, BACK ? -D : D, &w);
    Cx<R> v[3], u[9], o[3];
    in.load(n, v);
    U.load(MU, BACK ? n : s, u);
    apply_wraps(g, MU, w, v);
    if (BACK) su3_adj_mul_vec(u, v, o);
    else su3_mul_vec(u, v, o);
#pragma unroll
    for (int k = 0; k < 3; k++) acc[k] = acc[k] + f * o[k];
  }
  template <int DAG, int W, class Src>
  LMB_D void hop_w(const Geom &g, int s, const int *c, const Src &in, SmallHops<R> &sm) const {
    constexpr int MU = W >> 1, BACK = W & 1;
    int odd = 0;
#pragma unroll
    for (int d = 0; d < MU; d++) odd += c[d] + g.eta_off[d];
    const R sign = ((odd & 1) != 0) != (BACK != DAG) ? (R)-1 : (R)1;
    Cx<R> acc[3] = {Cx<R>(0, 0), Cx<R>(0, 0), Cx<R>(0, 0)};
    link_hop<MU, BACK, 1>(g, s, c, in, X, sign * fc, acc);
    if constexpr (NAIK) link_hop<MU, BACK, 3>(g, s, c, in, L, sign * lc, acc);
    put_hop(sm, W, 3, acc);
  }
  template <int DAG, int PH, class Src>
  LMB_D void hop(int w, const Geom &g, int s, const Src &in, SmallHops<R> &sm) const {
    int c[4];
    site_coords(g, s, c);
    switch (w) {
      case 0: hop_w<DAG, 0>(g, s, c, in, sm); break;
      case 1: hop_w<DAG, 1>(g, s, c, in, sm); break;
      case 2: hop_w<DAG, 2>(g, s, c, in, sm); break;
      case 3: hop_w<DAG, 3>(g, s, c, in, sm); break;
      case 4: hop_w<DAG, 4>(g, s, c, in, sm); break;
      case 5: hop_w<DAG, 5>(g, s, c, in, sm); break;
      case 6: hop_w<DAG, 6>(g, s, c, in, sm); break;
      default: hop_w<DAG, 7>(g, s, c, in, sm); break;
    }
  }
  template <int DAG, int PH, class Src>
  LMB_D void finish(int, const Geom &, int s, const Src &in, const SmallHops<R> &sm, Cx<R> *out) const {
    Cx<R> v[3];
    in.own(s, 0, v);
#pragma unroll
    for (int k = 0; k < 3; k++) {
      Cx<R> a = mass * v[k];
#pragma unroll
      for (int w = 0; w < 8; w++) a = a + get_hop(sm, w, k);
      out[k] = a;
    }
  }
};

// ---------------------------------------------------------------------------
// grid barrier with a sum: one counter of arrivals for the launch, and the
// blocks' partial sums in two alternating arrays (an array is written again
// only after the barrier in between, when all blocks have read it).  One
// thread per block polls the counter; a flag per block polled by every thread
// of every block, which saves the reading of the partial sums afterwards,
// measured slower from 128 blocks on (8^4: 2.48 against 1.68 ms a solve).
// ---------------------------------------------------------------------------
struct SmallGrid {
  unsigned *arrived;  // zeroed before the launch
  double *partials;   // 2 gridDim.x
};
constexpr int kSmallSpins = 1 << 21;  // about two seconds

LMB_D double small_block_sum(double x) {
  __shared__ double part[kSmallThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  __syncthreads();
  if (lane == 0) part[w] = x;
  __syncthreads();
  double t = 0;
#pragma unroll
  for (int i = 0; i < kSmallThreads / 32; i++) t += part[i];
  return t;
}

// the sum of x over the grid, added in the same order by every block.  False:
// some block did not arrive in time (the same answer for every thread of a
// block; blocks that wait for one that gave up give up as well)
template <bool SUM>
LMB_D bool small_grid_sum(const SmallGrid &gr, unsigned &epoch, double x, double &total) {
  __shared__ int met;
  if (SUM) x = small_block_sum(x);
  else __syncthreads();
  epoch++;
  double *part = gr.partials + (size_t)(epoch & 1) * gridDim.x;
  if (threadIdx.x == 0) {
    if (SUM) part[blockIdx.x] = x;
    __threadfence();
    atomicAdd(gr.arrived, 1u);
    const unsigned goal = epoch * gridDim.x;
    int n = 0;
    unsigned seen;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(gr.arrived) : "memory");
    } while (seen < goal && ++n < kSmallSpins);
    met = seen >= goal;
  }
  __syncthreads();
  if (!met) return false;
  if (SUM) {
    double t = 0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += kSmallThreads) t += __ldcg(part + b);
    total = small_block_sum(t);
  }
  return true;
}
LMB_D bool small_barrier(const SmallGrid &gr, unsigned &epoch) {
  double none;
  return small_grid_sum<false>(gr, epoch, 0.0, none);
}

// ---------------------------------------------------------------------------
// the iterations
// ---------------------------------------------------------------------------
// the passes of an application before its last: false when a barrier gave up
template <int DAG, int PS, class Op, class Src>
LMB_D bool small_first_passes(const Geom &g, const Op &op, const Src &in, SmallHops<typename Op::R> &hops,
                              float (*mag)[kSmallTile], const SmallGrid &gr, unsigned &epoch, int tiles, int64_t n) {
  if constexpr (Op::phases(DAG) > 1) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
      const int s = t * kSmallTile + lane;
      const bool site = s < n, mine = site && w < Op::NC / 3;
      if (site) op.template hop<DAG, 0>(w, g, s, in, hops);
      __syncthreads();
      Cx<typename Op::R> v[3];
      if (mine) op.template finish<DAG, 0>(w, g, s, in, hops, v);
      own_store(op.mid, s, w, mine, v, mag);
      __syncthreads();
    }
    return small_barrier(gr, epoch);
  }
  return true;
}

template <int PS, int PX, class Op>
__global__ void __launch_bounds__(kSmallThreads, small_min_blocks<PS>())
    small_cg_kernel(const Geom g, const Op op, const Field<PS, Op::NC> p, const Field<PS, Op::NC> r,
                    const Field<PS, Op::NC> tmp, const Field<PX, Op::NC> x, CGState *st, const SmallGrid gr,
                    const int iters) {
  typedef typename Op::R R;
  constexpr int NC = Op::NC, G = NC / 3, L0 = Op::phases(0) - 1, L1 = Op::phases(1) - 1;
  __shared__ SmallHops<R> hops;
  __shared__ float mag[G][kSmallTile];
  __shared__ CGState ls;
  if (threadIdx.x == 0) ls = *st;
  __syncthreads();
  if (ls.status != ST_RUNNING) return;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t n = op.sites(g);
  const int tiles = (int)((n + kSmallTile - 1) / kSmallTile);
  const SrcField<PS, NC> dir{p}, ap{tmp};
  unsigned epoch = 0;
  for (int it = 0; it < iters; it++) {
    double n2 = 0, total;
    if (!small_first_passes<0, PS>(g, op, dir, hops, mag, gr, epoch, tiles, n)) return;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {  // A
      const int s = t * kSmallTile + lane;
      const bool site = s < n, mine = site && w < G;
      if (site) op.template hop<0, L0>(w, g, s, dir, hops);
      __syncthreads();
      Cx<R> v[3];
      if (mine) {
        op.template finish<0, L0>(w, g, s, dir, hops, v);
#pragma unroll
        for (int k = 0; k < 3; k++) n2 += (double)norm2(v[k]);
      }
      own_store(tmp, s, w, mine, v, mag);
      __syncthreads();
    }
    if (!small_grid_sum<true>(gr, epoch, n2, total)) return;
    if (threadIdx.x == 0) finalize_pAp(&ls, total);
    __syncthreads();
    if (ls.status != ST_RUNNING) break;
    const R alpha = (R)ls.alpha;
    n2 = 0;
    if (!small_first_passes<1, PS>(g, op, ap, hops, mag, gr, epoch, tiles, n)) return;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {  // B
      const int s = t * kSmallTile + lane;
      const bool site = s < n, mine = site && w < G;
      if (site) op.template hop<1, L1>(w, g, s, ap, hops);
      __syncthreads();
      Cx<R> v[3], rv[3];
      if (mine) {
        Cx<R> pv[3], xv[3];
        own_load(p, s, w, pv);
        own_load(r, s, w, rv);
        own_load(x, s, w, xv);
        op.template finish<1, L1>(w, g, s, ap, hops, v);
#pragma unroll
        for (int k = 0; k < 3; k++) {
          rv[k] = rv[k] - alpha * v[k];
          xv[k] = xv[k] + alpha * pv[k];
          n2 += (double)norm2(rv[k]);
        }
        own_store(x, s, w, true, xv, mag);
      }
      own_store(r, s, w, mine, rv, mag);
      __syncthreads();
    }
    if (!small_grid_sum<true>(gr, epoch, n2, total)) return;
    if (threadIdx.x == 0) finalize_rr(&ls, total);
    __syncthreads();
    if (ls.status != ST_RUNNING) break;
    const R beta = (R)ls.beta;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {  // C
      const int s = t * kSmallTile + lane;
      const bool mine = s < n && w < G;
      Cx<R> pv[3], rv[3];
      if (mine) {
        own_load(p, s, w, pv);
        own_load(r, s, w, rv);
#pragma unroll
        for (int k = 0; k < 3; k++) pv[k] = rv[k] + beta * pv[k];
      }
      own_store(p, s, w, mine, pv, mag);
      if constexpr (PS == PREC_HALF && G > 1) __syncthreads();
    }
    if (!small_barrier(gr, epoch)) return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *st = ls;
}

}  // namespace lmb

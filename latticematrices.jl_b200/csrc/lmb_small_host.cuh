// lmb_small_host.cuh -- launch of the small-lattice solver (lmb_small.cuh).
#pragma once
#include "lmb_driver.cuh"
#include "lmb_small.cuh"

namespace lmb {

// resident blocks of a kernel of kSmallThreads threads per SM
inline int small_resident(const void *kern) {
  static std::mutex mu;
  static std::map<const void *, int> cache;
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(kern);
  if (it != cache.end()) return it->second;
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, kSmallThreads, 0) != cudaSuccess) n = 0;
  return cache[kern] = n;
}

template <int PS, int PX, class Op>
int small_cg(lmb_ctx *ctx, const Op &op, const Field<PS, Op::NC> &p, const Field<PS, Op::NC> &r,
             const Field<PS, Op::NC> &t, const Field<PX, Op::NC> &x, cudaStream_t st) {
  auto kern = small_cg_kernel<PS, PX, Op>;
  int64_t per_sm = limit_of(ctx, "blocks", INT64_MAX);  // set: assumed, not asked for
  if (per_sm == INT64_MAX) per_sm = small_resident((const void *)kern);
  const int64_t resident = per_sm * std::max(1, ctx->sm_count);
  // A phase of this kernel costs its barrier and as many tile latencies as a
  // block has tiles, a stage of the staged solver its launch and its longest
  // thread, then its bytes.  The line between them lies at a number of tiles
  // per resident block, which differs with how well the staged stencils of the
  // operator and storage use the chip.  Solves on 148 SMs, staged -> one
  // launch, on both sides of it:
  //   Wilson FP64 12^2x16^2 5.60 -> 5.29 ms, 16^4 7.84 -> 7.94; FP32 16^4 7.24
  //   -> 6.10; int16 12^4 4.74 -> 4.10, 12^2x16^2 5.31 -> 5.73.  Clover FP64
  //   12^4 9.33 -> 7.94, 12^2x16^2 12.0 -> 12.8; int16 8^2x12^2 7.97 -> 5.20,
  //   12^4 7.96 -> 8.02.  Staggered FP64 12^2x16^2 4.79 -> 3.97, 16^4 4.99 ->
  //   5.28; int16 16^4 5.44 -> 5.34.  HISQ FP64 12^4 2.85 -> 2.39, 12^2x16^2
  //   3.95 -> 4.03; FP32 12^2x16^2 4.05 -> 3.73; int16 12^4 3.25 -> 3.04,
  //   12^2x16^2 3.79 -> 4.82.  Even/odd clover 12^4 int16 4.99 -> 4.30,
  //   12^2x16^2 6.05 -> 7.23.  At 8^4: Wilson FP64 3.51 -> 1.68, clover int16
  //   6.27 -> 3.59, HISQ FP32 2.27 -> 1.43.
  const unsigned tiles = grid_for(op.sites(ctx->g), kSmallTile);
  if (resident < 1 || tiles > Op::kWaves * resident) return kNotSmall;
  // every block is resident (a cooperative launch): the barriers can be met
  const unsigned grid = (unsigned)std::min<int64_t>(tiles, resident);
  char *ws = (char *)workspace(ctx, "small_cg", 256 + 2 * sizeof(double) * resident);
  if (!ws) return kNotSmall;
  LMB_CUDA(ctx, cudaMemsetAsync(ws, 0, 256, st));
  Geom g = ctx->g;
  Op o = op;
  Field<PS, Op::NC> fp = p, fr = r, ft = t;
  Field<PX, Op::NC> fx = x;
  CGState *state = ctx->st_dev;
  SmallGrid gr{(unsigned *)ws, (double *)(ws + 256)};
  int iters = kSmallIters;
  void *args[] = {&g, &o, &fp, &fr, &ft, &fx, &state, &gr, &iters};
  const cudaError_t e = cudaLaunchCooperativeKernel((const void *)kern, dim3(grid), dim3(kSmallThreads), args, 0, st);
  // refused before anything ran: the device cannot hold the grid at once (a
  // process that was given a share of its SMs, say), or takes no such launch
  if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported || e == cudaErrorNotPermitted) {
    cudaGetLastError();
    return kNotSmall;
  }
  LMB_CUDA(ctx, e);
  return LMB_OK;
}

}  // namespace lmb

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
  // thread, then its bytes.  The line between them (kWaves) lies at a whole number
  // of tiles per resident block, which differs with how well the staged stencils
  // of the operator and storage use the chip.  Solves on 148 SMs (296 resident
  // blocks in FP64, 444 in FP32 and int16) by their tiles, staged -> one launch,
  // ms, the last size below each line | the first above it:
  //   Wilson FP64 1152 5.62 -> 5.27 | 2048 8.07 -> 7.87; FP32 2048 7.31 -> 6.21 |
  //     2560 8.18 -> 7.32; int16 882 5.17 -> 4.53 | 1152 5.34 -> 5.76
  //   clover FP64 882 11.0 -> 9.8 | 1152 12.1 -> 12.9; FP32 2048 15.0 -> 14.5 |
  //     2560 18.5 -> 17.7; int16 288 8.20 -> 5.27 | 648 8.07 -> 8.11
  //   staggered FP64 1152 4.73 -> 3.93 | 2048 5.10 -> 5.32; FP32 2048 5.38 -> 5.13 |
  //     2560 6.27 -> 6.61; int16 2048 5.62 -> 5.42 | 2560 6.76 -> 6.94
  //   HISQ FP64 882 3.24 -> 2.99 | 1152 3.95 -> 4.10; FP32 1152 4.12 -> 3.72 | 2048
  //     4.33 -> 4.92; int16 882 3.48 -> 3.50, 648 3.24 -> 3.07 | 1152 3.82 -> 4.84
  //   even/odd clover FP64 270 4.55 -> 3.40 | 315 4.80 -> 4.45; FP32 441 5.87 -> 4.55 |
  //     576 6.16 -> 6.46; int16 441 5.52 -> 4.90 | 576 5.92 -> 7.31; Wilson FP64 270
  //     2.73 -> 1.86 | 315 2.77 -> 2.30; FP32 441 3.66 -> 2.72 | 576 3.75 -> 3.58;
  //     int16 441 3.60 -> 2.91 | 576 3.74 -> 4.00
  //   domain wall FP64 288 8.03 -> 5.25 | 576 8.66 -> 8.23, 768 9.76 -> 10.9; FP32 432
  //     7.58 -> 5.91 | 576 7.86 -> 8.22; int16 432 7.92 -> 6.68 | 576 8.10 -> 9.65
  // (Sizes just above a line may still gain: a block more per wave is not worth a
  // line of its own.)
  const unsigned tiles = grid_for(op.sites(ctx->g), kSmallTile);
  int64_t waves = limit_of(ctx, "tiles", INT64_MAX);  // set: instead of the line
  if (waves == INT64_MAX) waves = Op::kWaves;
  if (resident < 1 || tiles > waves * resident) return kNotSmall;
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

// Instantiates and dispatches k_expert_rows for one weight type; included by the per-type .cu files with
// EXPERT_ROWS_QT set, so that the types compile side by side.
#pragma once

#include <algorithm>

#include "cuda_rt.h"
#include "expert_rows.cuh"

namespace moe {

template <int QT, int NMAT, int M, int G, int UPL, int FORM>
static cudaError_t launch_one(ExpertRowsArgs a, uint32_t max_groups, const uint32_t *grid_global, const LaunchCtx &ctx, cudaStream_t st) {
  constexpr bool q8k = act_is_q8k(QT);
  // With the row length known at compile time a CTA's eight warps take one batch of passes each; else the caller's count.
  constexpr uint32_t rpp = 32 / G;
  if (UPL > 0)
    a.rows_per_cta = 8 * rpp * rows_batch(NMAT, UPL, M, grid_words(QT) > 0);
  else if (a.rows_per_cta < 8 * rpp)
    a.rows_per_cta = 8 * rpp;
  const size_t smem = (size_t)M * act_row_stride(q8k, a.K) + 4 * grid_words(QT);
  auto kernel = k_expert_rows<QT, NMAT, M, G, UPL, FORM>;
  if (smem > 48 * 1024) {
    // The most a group's rows take, whatever this launch's row length: set once per device.
    static std::atomic<uint32_t> attr_done{0};
    const size_t most = (size_t)M * act_row_stride(q8k, kRowsMaxK) + 4 * grid_words(QT);
    if (smem > most) return cudaErrorInvalidValue;
    const cudaError_t e = ensure_dynamic_smem(kernel, most, attr_done, ctx.device);
    if (e != cudaSuccess) return e;
  }
  if (max_groups > 65535) return cudaErrorInvalidValue;  // the grid's second extent; the layer refuses such sizes at create
  // Slabs per CTA: four when that still leaves two CTAs for every CTA slot of the GPU (eight slots an SM), else two,
  // else one. Measured on 32 rows of Q8_0 (247 experts): gate/up 0.142 ms with one slab a CTA, 0.112 with four, 0.119 with eight.
  uint32_t slabs = 1;
  if (UPL > 0) {
    const uint64_t ctas = (uint64_t)((a.R + a.rows_per_cta - 1) / a.rows_per_cta) * max_groups, slots = 8ull * ctx.sms;
    slabs = ctas >= 4 * slots ? 4 : ctas >= 2 * slots ? 2 : 1;
    // CTAs that take the top-k for themselves first: no more than run at once (three an SM), eight slabs at most.
    if (FORM == ROWS_ROUTED) slabs = (uint32_t)std::min<uint64_t>(8, (ctas + 3 * ctx.sms - 1) / (3 * ctx.sms));
  }
  a.slabs = slabs;
  const dim3 grid((a.R + a.rows_per_cta * slabs - 1) / (a.rows_per_cta * slabs), max_groups, std::max(1u, a.halves));
  return launch_kernel(ctx.pdl, kernel, grid, dim3(256), smem, st, a, grid_global);
}

template <int QT, int NMAT, int M, int FORM>
static cudaError_t launch_shape(const ExpertRowsArgs &a, uint32_t max_groups, const uint32_t *grid_global, const LaunchCtx &ctx, cudaStream_t st) {
  // Lengths that the kernels are not specialised for take the general instantiation, which finds a row's units at run time.
  if (!rows_specialised(a.K)) return launch_one<QT, NMAT, M, 32, 0, FORM>(a, max_groups, grid_global, ctx, st);
  constexpr uint32_t kLong = kRowsLengths[0] / Unit<QT>::kValues, kMid = kRowsLengths[1] / Unit<QT>::kValues, kShort = kRowsLengths[2] / Unit<QT>::kValues;
  static_assert(sizeof(kRowsLengths) / sizeof(kRowsLengths[0]) == 3, "a form for each");
  if (a.K == kRowsLengths[0]) return launch_one<QT, NMAT, M, 32, kLong / 32, FORM>(a, max_groups, grid_global, ctx, st);
  // A row of 32 units (Q8_0's 512 values): 16 lanes with two units each, two rows a warp pass, so that a reduction and a
  // store serve twice the bytes.
  if (a.K == kRowsLengths[1]) return launch_one<QT, NMAT, M, (kMid < 32 ? kMid : 16), (kMid < 32 ? 1 : kMid / 16), FORM>(a, max_groups, grid_global, ctx, st);
  return launch_one<QT, NMAT, M, (kShort < 32 ? kShort : 32), 1, FORM>(a, max_groups, grid_global, ctx, st);
}

template <int QT, int NMAT>
cudaError_t launch_expert_rows(const ExpertRowsArgs &a, int M, uint32_t max_groups, const uint32_t *grid_global, const LaunchCtx &ctx, cudaStream_t st) {
  if constexpr (NMAT == 2) {
    if (a.route.rl && M == 1) return launch_shape<QT, NMAT, 1, ROWS_ROUTED>(a, max_groups, grid_global, ctx, st);
    if (a.route.rl && M == 2) return launch_shape<QT, NMAT, 2, ROWS_ROUTED>(a, max_groups, grid_global, ctx, st);
    if (a.route.rl) return cudaErrorInvalidValue;
  }
  if constexpr (NMAT == 1)
    if (a.act_f32) switch (M) {
        case 1: return launch_shape<QT, NMAT, 1, ROWS_QUANT>(a, max_groups, grid_global, ctx, st);
        case 2: return launch_shape<QT, NMAT, 2, ROWS_QUANT>(a, max_groups, grid_global, ctx, st);
        case 4: return launch_shape<QT, NMAT, 4, ROWS_QUANT>(a, max_groups, grid_global, ctx, st);
        case 8: return launch_shape<QT, NMAT, 8, ROWS_QUANT>(a, max_groups, grid_global, ctx, st);
        default: return cudaErrorInvalidValue;
      }
  switch (M) {
    case 1: return launch_shape<QT, NMAT, 1, ROWS_LISTED>(a, max_groups, grid_global, ctx, st);
    case 2: return launch_shape<QT, NMAT, 2, ROWS_LISTED>(a, max_groups, grid_global, ctx, st);
    case 4: return launch_shape<QT, NMAT, 4, ROWS_LISTED>(a, max_groups, grid_global, ctx, st);
    case 8: return launch_shape<QT, NMAT, 8, ROWS_LISTED>(a, max_groups, grid_global, ctx, st);
    default: return cudaErrorInvalidValue;
  }
}

template <int QT, int G, int UPL>
static cudaError_t launch_down_combine_one(DownCombineArgs a, const uint32_t *grid_global, const LaunchCtx &ctx, cudaStream_t st) {
  auto kernel = k_down_combine<QT, G, UPL>;
  const size_t smem = down_combine_smem(QT, a.T * a.used, a.K);
  if (smem > 48 * 1024) {
    static std::atomic<uint32_t> attr_done{0};
    const cudaError_t e = ensure_dynamic_smem(kernel, kDownCombineMaxSmem, attr_done, ctx.device);
    if (e != cudaSuccess) return e;
  }
  // One round of CTAs, two an SM: what a CTA does once (quantising the inner rows) is done no more often than that.
  a.rows_per_warp = (a.R + 16 * ctx.sms - 1) / (16 * ctx.sms);
  const dim3 grid((a.R + 8 * a.rows_per_warp - 1) / (8 * a.rows_per_warp));
  return launch_kernel(ctx.pdl, kernel, grid, dim3(256), smem, st, a, grid_global);
}

template <int QT>
cudaError_t launch_down_combine(const DownCombineArgs &a, const uint32_t *grid_global, const LaunchCtx &ctx, cudaStream_t st) {
  const uint32_t upr = a.K / Unit<QT>::kValues;
  if (a.T * a.used > kShortMax || a.T > kShortRows || down_combine_smem(QT, a.T * a.used, a.K) > kDownCombineMaxSmem) return cudaErrorInvalidValue;
  if (upr <= 8) return launch_down_combine_one<QT, 8, 1>(a, grid_global, ctx, st);
  if (upr <= 16) return launch_down_combine_one<QT, 16, 1>(a, grid_global, ctx, st);
  if (upr <= 32) return launch_down_combine_one<QT, 32, 1>(a, grid_global, ctx, st);
  if (upr <= 64) return launch_down_combine_one<QT, 32, 2>(a, grid_global, ctx, st);
  if (upr <= 128) return launch_down_combine_one<QT, 32, 4>(a, grid_global, ctx, st);
  return cudaErrorInvalidValue;
}
template cudaError_t launch_down_combine<EXPERT_ROWS_QT>(const DownCombineArgs &, const uint32_t *, const LaunchCtx &, cudaStream_t);

template cudaError_t launch_expert_rows<EXPERT_ROWS_QT, 1>(const ExpertRowsArgs &, int, uint32_t, const uint32_t *, const LaunchCtx &, cudaStream_t);
template cudaError_t launch_expert_rows<EXPERT_ROWS_QT, 2>(const ExpertRowsArgs &, int, uint32_t, const uint32_t *, const LaunchCtx &, cudaStream_t);

}  // namespace moe

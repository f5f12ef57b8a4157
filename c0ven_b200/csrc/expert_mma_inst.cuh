// Instantiates and launches k_expert_mma for one weight type; included by the per-type .cu files with EXPERT_MMA_QT set.
#pragma once

#include <algorithm>

#include "cuda_rt.h"
#include "expert_mma.cuh"

namespace moe {

template <int QT, int NMAT, int MOST>
static cudaError_t launch_mma_one(ExpertMmaArgs a, uint32_t max_entries, const LaunchCtx &ctx, cudaStream_t st) {
  auto kernel = k_expert_mma<QT, NMAT, MOST>;
  const size_t smem = mma_smem(QT, 8 * MOST, a.K);
  if (smem > 48 * 1024) {
    static std::atomic<uint32_t> attr_done{0};
    const cudaError_t e = ensure_dynamic_smem(kernel, kMmaMaxSmem, attr_done, ctx.device);
    if (e != cudaSuccess) return e;
  }
  // Slabs a CTA: rows are staged, and a codebook with them, once for all of them. Groups of up to eight rows come in their
  // hundreds: four slabs where that leaves an SM more CTAs than it runs at once (100 rows of Q8_0: 452 us with one slab
  // of gate and up and two of down, 410 with four). The list of short tiles, which holds a fraction of max_entries when
  // the routing is skewed, is cut finer, so that few experts still spread over the SMs (256 rows, skewed: 243 -> 200 us).
  const uint64_t ctas = (uint64_t)(a.R / kMmaCtaRows) * max_entries;
  a.slabs = MOST > 1 ? (NMAT == 2 ? 1 : 2) : ctas >= 16ull * ctx.sms ? 4 : ctas >= 8ull * ctx.sms ? 2 : 1;
  // The lists' lengths are the device's, often a fraction of max_entries: no more CTAs than four rounds of them, which then
  // take the entries in turn (CTAs that find their list ended cost some 3 ns each: 4,096 of them 10 us).
  const uint32_t gx = (a.R / kMmaCtaRows + a.slabs - 1) / a.slabs, most = std::max(1u, 8 * ctx.sms / gx);
  const dim3 grid(gx, std::min(max_entries, most));
  return launch_kernel(ctx.pdl, kernel, grid, dim3(256), smem, st, a);
}

template <int QT, int NMAT>
cudaError_t launch_expert_mma(const ExpertMmaArgs &a, uint32_t most_rows, uint32_t max_entries, const LaunchCtx &ctx, cudaStream_t st) {
  if (!mma_takes(QT, a.K, most_rows <= 8 ? 8 : kMmaRows) || a.R % kMmaCtaRows || most_rows > kMmaRows || max_entries == 0) return cudaErrorInvalidValue;
  return most_rows <= 8 ? launch_mma_one<QT, NMAT, 1>(a, max_entries, ctx, st) : launch_mma_one<QT, NMAT, 4>(a, max_entries, ctx, st);
}

template cudaError_t launch_expert_mma<EXPERT_MMA_QT, 1>(const ExpertMmaArgs &, uint32_t, uint32_t, const LaunchCtx &, cudaStream_t);
template cudaError_t launch_expert_mma<EXPERT_MMA_QT, 2>(const ExpertMmaArgs &, uint32_t, uint32_t, const LaunchCtx &, cudaStream_t);

}  // namespace moe

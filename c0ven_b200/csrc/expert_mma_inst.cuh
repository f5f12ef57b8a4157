// Instantiates and launches k_expert_mma for one weight type; included by the per-type .cu files with EXPERT_MMA_QT set.
#pragma once

#include "cuda_rt.h"
#include "expert_mma.cuh"

namespace moe {

template <int QT, int NMAT, int NT>
static cudaError_t launch_mma_one(ExpertMmaArgs a, uint32_t max_entries, const LaunchCtx &ctx, cudaStream_t st) {
  auto kernel = k_expert_mma<QT, NMAT, NT>;
  const size_t smem = mma_smem(QT, 8 * NT, a.K);
  if (smem > 48 * 1024) {
    static std::atomic<uint32_t> attr_done{0};
    const cudaError_t e = ensure_dynamic_smem(kernel, kMmaMaxSmem, attr_done, ctx.device);
    if (e != cudaSuccess) return e;
  }
  // Several slabs a CTA where that leaves every SM four CTAs and more: the rows are then staged once for all of them.
  const uint64_t ctas = (uint64_t)(a.R / kMmaCtaRows) * max_entries;
  a.slabs = ctas >= 16ull * ctx.sms ? 4 : ctas >= 8ull * ctx.sms ? 2 : 1;
  const dim3 grid((a.R / kMmaCtaRows + a.slabs - 1) / a.slabs, max_entries);
  return launch_kernel(ctx.pdl, kernel, grid, dim3(256), smem, st, a);
}

template <int QT, int NMAT>
cudaError_t launch_expert_mma(const ExpertMmaArgs &a, uint32_t most_rows, uint32_t max_entries, const LaunchCtx &ctx, cudaStream_t st) {
  if (!mma_takes(QT, a.K) || a.R % kMmaCtaRows || most_rows > kMmaRows || max_entries == 0 || max_entries > 65535) return cudaErrorInvalidValue;
  return most_rows <= 8 ? launch_mma_one<QT, NMAT, 1>(a, max_entries, ctx, st) : launch_mma_one<QT, NMAT, 2>(a, max_entries, ctx, st);
}

template cudaError_t launch_expert_mma<EXPERT_MMA_QT, 1>(const ExpertMmaArgs &, uint32_t, uint32_t, const LaunchCtx &, cudaStream_t);
template cudaError_t launch_expert_mma<EXPERT_MMA_QT, 2>(const ExpertMmaArgs &, uint32_t, uint32_t, const LaunchCtx &, cudaStream_t);

}  // namespace moe

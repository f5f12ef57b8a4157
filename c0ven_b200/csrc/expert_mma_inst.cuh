// Instantiates and launches k_expert_mma for one weight type; included by the per-type .cu files with EXPERT_MMA_QT set.
#pragma once

#include <algorithm>

#include "cuda_rt.h"
#include "expert_mma.cuh"

namespace moe {

template <int QT, int NMAT, int MOST>
static cudaError_t launch_mma_one(const ExpertMmaArgs &a, uint32_t max_entries, const LaunchCtx &ctx, cudaStream_t st) {
  auto kernel = k_expert_mma<QT, NMAT, MOST>;
  static std::atomic<uint32_t> attr_done{0};
  constexpr size_t kSmSmem = 228 * 1024, kMost = 227 * 1024;  // an SM's shared memory, 1 KB of it kept for every CTA; what a CTA can have
  const cudaError_t e = ensure_dynamic_smem(kernel, kMost, attr_done, ctx.device);
  if (e != cudaSuccess) return e;
  auto smem_of = [&](uint32_t warps) {
    return (size_t)mma_smem(QT, 8 * MOST, a.K) + (size_t)warps * mma_stages(QT, MOST) * Frag<QT>::kStage;
  };
  // Sixteen warps an SM, in two CTAs; in one where two CTAs' rows do not fit (32 rows of 2,560 values).
  uint32_t warps = 8, per_sm = MOST == 1 && grid_words(QT) ? 3 : 2;
  while (per_sm > 1 && per_sm * (smem_of(8) + 1024) > kSmSmem) per_sm--;
  if (per_sm == 1 && 32 * 16 <= mma_threads(MOST) && smem_of(16) <= kMost) warps = 16;
  // Gate and up: an item is some 16 to 32 stages a warp, so CTAs of one item each, up to eight rounds of them, are shared out by
  // the SMs as they come free. A down item is a stage or four: one round of CTAs, each with runs of items. (One round and eight,
  // layer: Q8_0 60 rows 301 and 274 us, Q4_K 777 rows 384 and 377 for gate and up; 100 rows of Q4_K 242 and 252 for down.) CTAs past
  // the items cost some 4 us a thousand: sixteen rounds lose that again (Q4_K 32 rows 168 -> 188).
  constexpr uint32_t kRounds = NMAT == 1 ? 1 : 8;
  const uint64_t items = (uint64_t)(a.R / (16 * warps)) * max_entries;
  const dim3 grid((unsigned)std::min<uint64_t>(items, (uint64_t)kRounds * per_sm * ctx.sms));
  return launch_kernel(ctx.pdl, kernel, grid, dim3(32 * warps), smem_of(warps), st, a);
}

template <int QT, int NMAT>
cudaError_t launch_expert_mma(const ExpertMmaArgs &a, uint32_t most_rows, uint32_t max_entries, const LaunchCtx &ctx, cudaStream_t st) {
  if (!mma_takes(QT, a.K, most_rows <= 8 ? 8 : kMmaRows) || a.R % kMmaRowsUnit || most_rows > kMmaRows || max_entries == 0) return cudaErrorInvalidValue;
  return most_rows <= 8 ? launch_mma_one<QT, NMAT, 1>(a, max_entries, ctx, st) : launch_mma_one<QT, NMAT, 4>(a, max_entries, ctx, st);
}

template cudaError_t launch_expert_mma<EXPERT_MMA_QT, 1>(const ExpertMmaArgs &, uint32_t, uint32_t, const LaunchCtx &, cudaStream_t);
template cudaError_t launch_expert_mma<EXPERT_MMA_QT, 2>(const ExpertMmaArgs &, uint32_t, uint32_t, const LaunchCtx &, cudaStream_t);

}  // namespace moe

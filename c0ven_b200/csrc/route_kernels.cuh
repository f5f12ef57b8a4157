// The block's routing and elementwise stages: activation quantisers, router logits, top-k with renormalised weights,
// the stable pack into expert order with its tiles and groups, and the weighted combine. They replace the reference's
// quantize_a8 (kernels/include/a8.h:9-16), the router product (kernels/common.cl:114-158, kernels/gemm.cl:51-115),
// router / p_router (kernels/models/qwen4exp/layer.cl:765-847, prompt.cl:652-678, route.h:39-98), p_moe_count / scan /
// fill (prompt.cl:682-738), moe_group (layer.cl:894-978) and moe_combine / p_moe_combine (layer.cl:869-883,
// prompt.cl:769-786).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "expert_rows.cuh"
#include "expert_tiles.cuh"
#include "quant_rows.cuh"
#include "router_topk.cuh"

namespace moe {

constexpr uint32_t kTileRows = 64;      // MOE_TILE (shared/moe_tile.h:9)
constexpr uint32_t kChunkTokens = 32;   // rows one CTA of the top-k kernel routes: a chunk of the pack

// ---------------------------------------------------------------------------------------------------------------
// Activation quantisers. One warp per 256 values.

// With gate set (a vector of `per_row` * 256 floats), a block of 256 values also leaves its part of the row's product
// with the vector in gate_parts[block]: the shared expert's gate logit, summed by the top-k kernel.
__device__ __forceinline__ void gate_part(const float4 &a, const float4 &b, const float *gate, uint32_t per_row, uint64_t blk,
                                          uint32_t lane, float *gate_parts) {
  const float4 *g = (const float4 *)(gate + (blk % per_row) * 256);
  const float4 ga = g[2 * lane], gb = g[2 * lane + 1];
  float s = a.x * ga.x + a.y * ga.y + a.z * ga.z + a.w * ga.w + b.x * gb.x + b.y * gb.y + b.z * gb.z + b.w * gb.w;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if (lane == 0) gate_parts[blk] = s;
}

// What the tensor-core router product takes of a row (steps of many rows): x as the sum of two f16 numbers, hi = f16(x)
// and lo = f16(x - hi), 22 bits of x between them, and the block's sum of squares, from which the top-k kernel bounds
// that product's error for the row.
struct RouterSplit {
  __half *hi, *lo;     // [rows][K] each; null: not wanted
  float *norm2_parts;  // [rows][K / 256]
};
__device__ __forceinline__ uint32_t split_pair(float x0, float x1, uint32_t &lo) {
  const __half2 h = __floats2half2_rn(x0, x1);
  const float2 hf = __half22float2(h);
  const __half2 l = __floats2half2_rn(x0 - hf.x, x1 - hf.y);
  lo = *(const uint32_t *)&l;
  return *(const uint32_t *)&h;
}
__device__ __forceinline__ void router_split(const float4 &a, const float4 &b, uint64_t blk, uint32_t lane, const RouterSplit &rs) {
  uint4 hi, lo;
  hi.x = split_pair(a.x, a.y, lo.x), hi.y = split_pair(a.z, a.w, lo.y);
  hi.z = split_pair(b.x, b.y, lo.z), hi.w = split_pair(b.z, b.w, lo.w);
  ((uint4 *)(rs.hi + blk * 256))[lane] = hi;
  ((uint4 *)(rs.lo + blk * 256))[lane] = lo;
  float s = a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w + b.x * b.x + b.y * b.y + b.z * b.z + b.w * b.w;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if (lane == 0) rs.norm2_parts[blk] = s;
}

// BOTH: the rows in the other form too (job2): one reading of them for the two.
template <bool Q8K, bool BOTH>
static __global__ void __launch_bounds__(256) k_quant(const float *x, uint64_t nblk256, const QuantJob job, const float *__restrict__ gate,
                                              uint32_t per_row, float *__restrict__ gate_parts, RouterSplit rs, const QuantJob job2) {
  dependents_may_launch(), wait_for_predecessors();
  const uint64_t blk = (uint64_t)blockIdx.x * 8 + threadIdx.x / 32;
  if (blk >= nblk256) return;
  const uint32_t lane = threadIdx.x % 32;
  const float4 a = ((const float4 *)(x + blk * 256))[2 * lane], b = ((const float4 *)(x + blk * 256))[2 * lane + 1];
  if (gate) gate_part(a, b, gate, per_row, blk, lane, gate_parts);
  if (rs.hi) router_split(a, b, blk, lane, rs);
  quantize_store<Q8K>(a, b, blk, lane, job);
  if constexpr (BOTH) quantize_store<!Q8K>(a, b, blk, lane, job2);
}

// ---------------------------------------------------------------------------------------------------------------
// Router logits: rl[t][e] = W[e] . x[t] for the NE experts and, as row NE, the shared expert's gate vector. Every
// product is summed in kRouterPieces equal pieces of the row, each a chain of fused multiply-adds from 0 in index
// order, the pieces then added in order, and an expert's bias last. Both kernels and the CPU oracle keep this one
// order, so that the logits, and with them the chosen experts, agree bit for bit whatever the row count.

// A CTA takes four of the router's rows and up to ROWS rows of x: a warp a piece, its lanes the pairs of a row of x and one of the
// router's (8 rows: a chain a lane) or a row of x each (32 rows: four chains a lane). Both come through a ring in shared memory by
// 16-byte asynchronous copies, 16 values of every piece a stage, so that each of the router's rows is read from HBM once. What bounds
// it is the chain of its stages, sixteen at 2,048 values, each a wait for its copies and a barrier: no unit is near its limit (32
// rows, ncu: issue slots 29 % and the L1 39 % busy while an SM has work). (A lane walking its
// piece of a weight row itself for two rows of x a CTA, the router's 4 MB read out of L2 again for every two rows: 33 us at 32
// rows by ncu, cold, 18 to 20 now; two layers of 32 rows of IQ3_S 6 % less, 64 rows of Q8_0 377 and 272 together with the groups'
// other kernel, four rows of Q4_K with Q6_K 70 and 64.)
// One row has a kernel of its own, k_router_logits_one: by the form for 8 rows, with rings of 42 to 104 KB, which keep the next
// kernel's waiting CTAs off the SM, the layer in Q8_0 took 27.5 to 28.8 us, 26.7 so.
// The step's quantisers ride along: the first sq.ctas CTAs of every grid row share out the blocks of x among their warps,
// so that quantising x is neither a launch of its own in front of the router nor behind it. A warp takes as many blocks as
// that leaves it.
struct StepQuant {
  QuantJob job[2];  // the routed experts' form of x, and the shared expert's where it is another one
  uint64_t nblk;
  uint32_t ctas;    // in the grid's first extent; 0: x is quantised elsewhere
};
__device__ __forceinline__ void quantize_share(const float *x, const StepQuant &sq) {
  wait_for_predecessors();
  const uint32_t lane = threadIdx.x % 32, warps = blockDim.x / 32;
  const uint64_t step = (uint64_t)gridDim.y * sq.ctas * warps;
  for (uint64_t blk = ((uint64_t)blockIdx.y * sq.ctas + blockIdx.x) * warps + threadIdx.x / 32; blk < sq.nblk; blk += step) {
    const float4 a = ((const float4 *)(x + blk * 256))[2 * lane], b = ((const float4 *)(x + blk * 256))[2 * lane + 1];
#pragma unroll
    for (int j = 0; j < 2; j++) {
      if (!sq.job[j].q) continue;
      if (sq.job[j].q8k)
        quantize_store<true>(a, b, blk, lane, sq.job[j]);
      else
        quantize_store<false>(a, b, blk, lane, sq.job[j]);
    }
  }
}
constexpr uint32_t kRouterExperts = 4;                     // the router's rows a CTA takes
constexpr uint32_t kRouterFewRows = 8, kRouterRows = 32;   // rows of x a CTA takes: the two forms
constexpr uint32_t kRouterChunk = 16;                      // values of a piece a stage holds
constexpr uint32_t kRouterXRow = kRouterChunk * 4 + 16;    // bytes from a row's chunk to the next: spreads a quarter-warp over the banks
constexpr uint32_t kRouterWBytes = kRouterExperts * kRouterPieces * kRouterChunk * 4;
__host__ __device__ constexpr uint32_t router_ring(uint32_t rows) { return rows == kRouterFewRows ? 6 : 4; }
__host__ __device__ constexpr uint32_t router_x_bytes(uint32_t rows) { return kRouterPieces * rows * kRouterXRow; }
__host__ __device__ constexpr uint32_t router_rows_smem(uint32_t rows) { return router_ring(rows) * (router_x_bytes(rows) + kRouterWBytes); }  // 42, 88 KB
template <uint32_t ROWS>
static __global__ void __launch_bounds__(32 * kRouterPieces) k_router_logits_rows(const float *x, uint32_t T, uint32_t E,
                                                          const float *__restrict__ W, uint32_t N,
                                                          const float *__restrict__ bias, uint32_t NE,
                                                          float *__restrict__ rl, const StepQuant sq) {
  extern __shared__ __align__(16) uint8_t smem[];
  dependents_may_launch();
  const uint32_t tid = threadIdx.x, lane = tid % 32, piece_of = tid / 32;
  if (blockIdx.x < sq.ctas) return quantize_share(x, sq);
  constexpr uint32_t S = router_ring(ROWS), C = kRouterChunk, kXBytes = router_x_bytes(ROWS), kStage = kXBytes + kRouterWBytes;
  constexpr uint32_t CHAINS = kRouterExperts * ROWS / 32;  // a lane's
  const uint32_t piece = E / kRouterPieces, nch = piece / C;
  const uint32_t t0 = blockIdx.y * ROWS, tn = min(ROWS, T - t0), e0 = (blockIdx.x - sq.ctas) * kRouterExperts;
  const uint32_t smem32 = (uint32_t)__cvta_generic_to_shared(smem);
  // Four neighbouring threads bring a piece's 64 bytes of a row: the router's rows by half of the threads, x's by all of them.
  const uint32_t part = tid % 4, pc = tid / 4 % kRouterPieces, first = tid / 32;
  auto ask_w = [&](uint32_t c) {
    if (first < kRouterExperts)
      cp_async16(smem32 + c % S * kStage + kXBytes + (first * kRouterPieces + pc) * (C * 4) + part * 16,
                 W + (uint64_t)min(e0 + first, N - 1) * E + pc * piece + c * C + part * 4);
  };
  auto ask_x = [&](uint32_t c) {
    for (uint32_t t = first; t < tn; t += 8)
      cp_async16(smem32 + c % S * kStage + (pc * ROWS + t) * kRouterXRow + part * 16, x + (uint64_t)(t0 + t) * E + pc * piece + c * C + part * 4);
  };
  auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
  // The first weights are on their way before the rows are there: they are nobody's output.
#pragma unroll
  for (uint32_t c = 0; c + 1 < S; c++)
    if (c < nch) ask_w(c);
  wait_for_predecessors();
#pragma unroll
  for (uint32_t c = 0; c + 1 < S; c++) {
    if (c < nch) ask_x(c);
    commit();
  }
  const uint32_t my_row = lane % ROWS, my_first = lane / ROWS;
  float p[CHAINS];
#pragma unroll
  for (uint32_t e = 0; e < CHAINS; e++) p[e] = 0.0f;
  for (uint32_t c = 0; c < nch; c++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
    __syncthreads();  // every thread's copies of this chunk are there, and the stage asked for next has been read
    if (c + S - 1 < nch) ask_w(c + S - 1), ask_x(c + S - 1);
    commit();
    const uint8_t *st = smem + c % S * kStage;
    const float4 *xs = (const float4 *)(st + (piece_of * ROWS + my_row) * kRouterXRow);
    const float4 *ws = (const float4 *)(st + kXBytes + (my_first * kRouterPieces + piece_of) * (C * 4));
#pragma unroll
    for (uint32_t i = 0; i < C / 4; i++) {
      const float4 xv = xs[i];
#pragma unroll
      for (uint32_t e = 0; e < CHAINS; e++) {
        const float4 wv = ws[e * kRouterPieces * (C / 4) + i];
        p[e] = fmaf(xv.x, wv.x, p[e]);
        p[e] = fmaf(xv.y, wv.y, p[e]);
        p[e] = fmaf(xv.z, wv.z, p[e]);
        p[e] = fmaf(xv.w, wv.w, p[e]);
      }
    }
  }
  // The pieces of a logit added in order, a thread a logit.
  __syncthreads();
  float *sum = (float *)smem;  // [expert][piece][row]
#pragma unroll
  for (uint32_t e = 0; e < CHAINS; e++) sum[((my_first + e) * kRouterPieces + piece_of) * ROWS + my_row] = p[e];
  __syncthreads();
  const uint32_t e = tid % kRouterExperts, t = tid / kRouterExperts, row = e0 + e;
  if (t < tn && row < N) {
    float tot = sum[e * kRouterPieces * ROWS + t];
#pragma unroll
    for (uint32_t j = 1; j < kRouterPieces; j++) tot = __fadd_rn(tot, sum[(e * kRouterPieces + j) * ROWS + t]);
    if (bias && row < NE) tot = __fadd_rn(tot, bias[row]);
    rl[(uint64_t)(t0 + t) * N + row] = tot;
  }
}

// One row: a warp takes four of the router's rows, 8 lanes a row, lane s walking piece s of it with D loads of 16 bytes in flight (a
// piece is a multiple of 4 D values: 8 always, 16 when the piece is a multiple of 64 values); x in shared memory. A CTA is a warp.
template <int D>
static __global__ void __launch_bounds__(32) k_router_logits_one(const float *x, uint32_t E, const float *__restrict__ W, uint32_t N,
                                                         const float *__restrict__ bias, uint32_t NE, float *__restrict__ rl, const StepQuant sq) {
  extern __shared__ __align__(16) float xs[];  // each piece padded by 4 floats to spread the banks
  dependents_may_launch();
  if (blockIdx.x < sq.ctas) return quantize_share(x, sq);
  const uint32_t piece = E / kRouterPieces, pstride = piece + 4;
  const uint32_t lane = threadIdx.x, s = lane % 8, row = (blockIdx.x - sq.ctas) * 4 + lane / 8;
  // The first weights are on their way while the row is staged (and before it is there: the weights are nobody's output).
  const float4 *w = (const float4 *)(W + (uint64_t)min(row, N - 1) * E + s * piece);
  float4 wq[D];
#pragma unroll
  for (int i = 0; i < D; i++) wq[i] = __ldg(w + i);
  wait_for_predecessors();
  for (uint32_t k4 = lane; k4 < E / 4; k4 += 32) *(float4 *)(xs + 4 * k4 / piece * pstride + 4 * k4 % piece) = ((const float4 *)x)[k4];
  __syncwarp();
  float p = 0.0f;
  const float *xp = xs + s * pstride;
  for (uint32_t i0 = 0; i0 < piece / 4; i0 += D) {
    float4 cur[D];
#pragma unroll
    for (int i = 0; i < D; i++) cur[i] = wq[i];
    if (i0 + D < piece / 4) {
#pragma unroll
      for (int i = 0; i < D; i++) wq[i] = __ldg(w + i0 + D + i);
    }
#pragma unroll
    for (int i = 0; i < D; i++) {
      const float4 xv = *(const float4 *)(xp + 4 * (i0 + i));
      p = fmaf(xv.x, cur[i].x, p);
      p = fmaf(xv.y, cur[i].y, p);
      p = fmaf(xv.z, cur[i].z, p);
      p = fmaf(xv.w, cur[i].w, p);
    }
  }
  float tot = __shfl_sync(0xffffffffu, p, lane & ~7u);
#pragma unroll
  for (int j = 1; j < (int)kRouterPieces; j++) tot = __fadd_rn(tot, __shfl_sync(0xffffffffu, p, (lane & ~7u) + j));
  if (s == 0 && row < N) {
    if (bias && row < NE) tot = __fadd_rn(tot, bias[row]);
    rl[row] = tot;
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Top-k kernels over router_topk.cuh.
// The block's part: its rows' ids, weights and gates written, the chunk's count of every expert left in hist (shared,
// 512 words) and, when s_ids is not null, the chunk's ids there too (shared, kChunkTokens * K words). hist null: the
// caller counts the chunks' experts itself (k_chunk_hist), and the block may be of any number of warps. ex_smem:
// kExWarpBytes of shared memory for every warp of the block, or null.
__device__ __forceinline__ void router_topk_block(const float *rl, const RouterApprox ap, const float *__restrict__ bias,
                                                  uint32_t T, uint32_t NE, uint32_t K, int32_t *__restrict__ ids, float *__restrict__ w,
                                                  float *__restrict__ gs, uint32_t *hist, int32_t *s_ids, uint8_t *ex_smem = nullptr) {
  if (hist) {
    for (uint32_t i = threadIdx.x; i < NE; i += blockDim.x) hist[i] = 0;
    __syncthreads();
  }
  const uint32_t warp = threadIdx.x / 32, t = blockIdx.x * (blockDim.x / 32) + warp;
  if (t < T)
    router_topk_row(t, rl, ap, bias, NE, K, ids, w, gs, hist, s_ids ? s_ids + warp * K : nullptr, ex_smem ? ex_smem + warp * kExWarpBytes : nullptr);
  if (hist) __syncthreads();
}

// The top-k alone, a few rows a CTA and no barrier in it: for long steps, whose rows wait on memory for their exact
// recomputations (with many small CTAs an SM always has rows that are not waiting, and no row waits for the slowest of its
// chunk), and for exact logits where the step's rows are more than one CTA's warps should take one after another. The
// chunks' counts then come from k_chunk_hist.
constexpr uint32_t kTopkRowsPerCta = 4;
static __global__ void __launch_bounds__(32 * kTopkRowsPerCta) k_router_topk_rows(const float *rl, const RouterApprox ap, const float *__restrict__ bias, uint32_t T,
                                                                                 uint32_t NE, uint32_t K, int32_t *__restrict__ ids,
                                                                                 float *__restrict__ w, float *__restrict__ gs) {
  __shared__ __align__(16) uint8_t ex_smem[kTopkRowsPerCta * kExWarpBytes];
  dependents_may_launch(), wait_for_predecessors();
  router_topk_block(rl, ap, bias, T, NE, K, ids, w, gs, nullptr, nullptr, ap.E % (kRouterPieces * kExChunk) == 0 ? ex_smem : nullptr);
}

static __global__ void __launch_bounds__(32 * kChunkTokens) k_router_topk(const float *__restrict__ rl, const RouterApprox ap,
                                                                  const float *__restrict__ bias, uint32_t T, uint32_t NE,
                                                                  uint32_t K, int32_t *__restrict__ ids,
                                                                  float *__restrict__ w, float *__restrict__ gs,
                                                                  uint32_t *__restrict__ chunk_hist) {
  __shared__ uint32_t hist[512];
  router_topk_block(rl, ap, bias, T, NE, K, ids, w, gs, hist, nullptr);
  for (uint32_t i = threadIdx.x; i < NE; i += blockDim.x) chunk_hist[(uint64_t)blockIdx.x * NE + i] = hist[i];
}

// The same counts for expert ids that come from elsewhere (the rows another GPU sent): chunk c holds entries
// [c * chunk_len, (c + 1) * chunk_len) of ids.
static __global__ void __launch_bounds__(256) k_chunk_hist(const int32_t *ids, uint32_t A, uint32_t chunk_len,
                                                   uint32_t NE, uint32_t first_expert, uint32_t *__restrict__ chunk_hist) {
  __shared__ uint32_t hist[512];
  dependents_may_launch(), wait_for_predecessors();
  for (uint32_t i = threadIdx.x; i < NE; i += blockDim.x) hist[i] = 0;
  __syncthreads();
  const uint32_t a0 = blockIdx.x * chunk_len, a1 = min(A, a0 + chunk_len);
  for (uint32_t a = a0 + threadIdx.x; a < a1; a += blockDim.x) {
    const uint32_t e = (uint32_t)ids[a] - first_expert;
    if (e < NE) atomicAdd(&hist[e], 1u);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < NE; i += blockDim.x) chunk_hist[(uint64_t)blockIdx.x * NE + i] = hist[i];
}

// The expert of every row a GPU receives in the rows' all-to-all: the sources one after another, each source's rows in
// expert order. cnt_all [world][NE] is every GPU's rows per expert; this GPU owns experts first .. first + per. Block
// b = source * per + local expert sums the runs before its own and fills its run.
static __global__ void __launch_bounds__(128) k_received_ids(const uint32_t *__restrict__ cnt_all, uint32_t NE, uint32_t first, uint32_t per,
                                                     int32_t *__restrict__ ids) {
  __shared__ uint32_t part[128];
  const uint32_t b = blockIdx.x;
  uint32_t sum = 0;
  for (uint32_t p = threadIdx.x; p < b; p += 128) sum += cnt_all[(uint64_t)(p / per) * NE + first + p % per];
  part[threadIdx.x] = sum;
  __syncthreads();
  for (uint32_t off = 64; off; off >>= 1) {
    if (threadIdx.x < off) part[threadIdx.x] += part[threadIdx.x + off];
    __syncthreads();
  }
  const uint32_t start = part[0], n = cnt_all[(uint64_t)(b / per) * NE + first + b % per];
  for (uint32_t i = threadIdx.x; i < n; i += 128) ids[start + i] = (int32_t)(first + b % per);
}

// The rows' f16 activations put in expert order, so that the tile kernels' bulk-tensor copies find a tile's rows one
// after another (the reference's p_moe_scatter, kernels/models/qwen4exp/prompt.cl:744-754), for a step whose every row has
// `per_row` places in expert order, place_of[t * per_row + k]: dst[place_of[t * per_row + k]] = src[t]. A CTA a row; a
// thread reads 16 bytes of it once and writes them per_row times. (The same copy taken from the places' side, dst[r] =
// src[row_src[r]], reads a row once per place, in expert order, long after its last use left the L2: at 32,768 rows
// of 2,048 values and ten places a row it read 1.0 GB from DRAM for the 134 MB of rows there are, and took twice as long.)
static __global__ void __launch_bounds__(256) k_scatter_f16(const __half *src, const uint32_t *place_of, uint32_t per_row,
                                                    uint32_t K, __half *__restrict__ dst, const uint32_t *ntiles) {
  dependents_may_launch(), wait_for_predecessors();
  if (*ntiles == 0) return;  // a short step none of whose experts goes to the tile kernels
  const uint64_t t = blockIdx.x;
  __shared__ uint32_t places[16];  // n_used at most
  if (threadIdx.x < per_row) places[threadIdx.x] = place_of[t * per_row + threadIdx.x];
  __syncthreads();
  for (uint32_t c = threadIdx.x; c < K / 8; c += 256) {
    const uint4 v = ((const uint4 *)(src + t * K))[c];
    for (uint32_t k = 0; k < per_row; k++) ((uint4 *)(dst + (uint64_t)places[k] * K))[c] = v;
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Pack. Assignments a = t * K + k go into expert order by a stable counting sort: experts ascending, and inside an
// expert's run ascending a. The reference's fill takes rows by atomic increments, so its order inside a run depends on
// scheduling (prompt.cl:730-737); this one has no atomics on the order and gives the same permutation every time.

// Whether an expert with n rows goes to the tensor-core kernels (tensor_min 0: none does).
__host__ __device__ inline bool n_is_tensor(uint32_t n, uint32_t tensor_min) { return tensor_min != 0 && n >= tensor_min; }

// One CTA of 512 threads, thread e for expert e: sums the chunks' counts, scans them over the experts, writes tiles
// and groups. first_expert: the id of slot 0. group_max: the most rows a group holds (<= kGroupMax). tensor_budget, when
// not 0, lets the step lower tensor_min itself: to the least of 1, 2, 4, 8 rows that sends at most tensor_budget experts
// to the tile kernels. With skewed routing a short step has a few experts with many rows, which the tile kernels take
// in the time the integer-dot kernel needs for one of them; with even routing it has hundreds of experts with one or
// two rows, whose tiles would be all decode and no product: the threshold moves only if the experts that then change
// kernels hold at least half of the step's rows.
// The scan itself, for every thread of a CTA of 512 threads or more (the threads past 511 only keep the barriers):
// thread e < NE brings its expert's row count `run`; returns the first row of the expert's run. One CTA works while the
// step waits, so what counts is its chain of barriers and dependent reads: prefix sums by shuffles with one barrier
// between the warps' part and the block's, and the short tiles ranked by a counting sort over their lengths (every
// thread reading all 512 lengths to find its rank took longer than all the rest).
__device__ __forceinline__ uint32_t pack_scan_block(uint32_t e, uint32_t run, uint32_t NE, uint32_t first_expert, uint32_t tensor_min,
                                                    uint32_t tensor_budget, uint32_t group_max, const PackOut &o) {
  constexpr uint32_t kWarps = 16, kSums = 8;
  __shared__ uint32_t s_sum[kSums][kWarps], s_ge[4][kWarps], s_rows_ge[4][kWarps];
  __shared__ uint16_t s_len[kWarps][kTileN];  // short tiles of a length in a warp; then how many of that length come before the warp's
  __shared__ uint32_t s_bin[kTileN / 32];
  const bool in = e < 512;
  const uint32_t lane = e % 32, warp = e / 32;
  if (!in || e >= NE) run = 0;
  // A value over the 16 warps' entries of a row: the sum before this warp's, and the sum of all.
  auto before_and_all = [&](const uint32_t *row, uint32_t &all) {
    uint32_t v = lane < kWarps ? row[lane] : 0;
    const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? v : 0);
    all = __reduce_add_sync(0xffffffffu, v);
    return before;
  };
  if (tensor_budget) {
    // Lower only if the experts that would move hold at least half of the step's rows: moving a few rows costs two
    // more kernels for nothing.
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t least = 1u << j, c = __popc(__ballot_sync(0xffffffffu, run >= least));
      const uint32_t r = __reduce_add_sync(0xffffffffu, run >= least ? run : 0);
      if (in && lane == 0) s_ge[j][warp] = c, s_rows_ge[j][warp] = r;
    }
    __syncthreads();
    uint32_t ge[4], rows_ge[4];
#pragma unroll
    for (int j = 0; j < 4; j++) before_and_all(s_ge[j], ge[j]), before_and_all(s_rows_ge[j], rows_ge[j]);
    if (ge[0] <= tensor_budget) {
      tensor_min = 1;  // few experts in all: every one to the tile kernels
    } else {
      const int pick = ge[1] <= tensor_budget ? 1 : ge[2] <= tensor_budget ? 2 : ge[3] <= tensor_budget ? 3 : 0;
      if (pick > 0 && 2 * (pick == 1 ? rows_ge[1] : pick == 2 ? rows_ge[2] : rows_ge[3]) >= rows_ge[0]) tensor_min = min(tensor_min, 1u << pick);
    }
  }
  const bool tensor = n_is_tensor(run, tensor_min);
  // Rows up to which an expert with one short tile goes to the few-rows kernel. That kernel takes 16 weight rows a warp
  // for as long as the row is, and longer with every eight activation rows, so it needs many warps: a step that hits 80
  // experts (256 rows, skewed) was slower with experts of 32 rows there (243 us) than of 16 (231), one that hits 512
  // (777 rows) faster (463 against 564). In a step that few experts share (FEW_IF_ALL: below 1,280 assignments) it wins
  // where all have a few rows (13 rows over 73 experts in IQ2_S: 239 -> 187 us) and loses beside the tile kernels, which
  // take a long expert in the time of a short one (64 rows, skewed: 217 -> 258).
  uint32_t few = 0;
  if (o.few_rows == FEW_BY_ROWS) {
    few = __syncthreads_count(run > 0) < 256 ? 16 : 32;
  } else if (o.few_rows == FEW_IF_ALL) {
    few = __syncthreads_or(tensor && run > 8) ? 0 : 8;
  }
  const uint32_t n = run, nt = (n + kTileRows - 1) / kTileRows, ng = tensor ? 0 : (n + group_max - 1) / group_max;
  const uint32_t nb = tensor ? (n + kTileN - 1) / kTileN : 0;
  // Big tiles, in the order the tile kernels deal them to their CTAs round by round. First the experts that have at
  // least one full tile of kTileN rows, in expert order, each one's tiles side by side, its last, shorter one too: the
  // CTAs that take them run at the same time, so an expert's weights come from HBM once and from L2 after that (with
  // the short tiles all at the end, as this list once had them, every expert's weights were read from HBM again for
  // its short tile: 3.5 GB of traffic a 32,768-row gate/up launch against 2.6 GB the algorithm needs). Then the experts
  // with one short tile only, by falling row count (ties in expert order), so that the last rounds hold the
  // shortest items.
  const uint32_t nfull = tensor ? n / kTileN : 0, rem = tensor ? n % kTileN : 0;
  const uint32_t mine = nfull ? nfull + (rem != 0) : 0, len = nfull ? 0 : rem;  // len: the expert's short tile, 0 without one
  // Inclusive sums within the warp of what the lists are laid out by; plain sums of the rest.
  uint32_t v[4] = {n, nt, ng, mine};
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (uint32_t off = 1; off < 32; off <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, v[j], off);
      if (lane >= off) v[j] += u;
    }
  const uint32_t hit = __popc(__ballot_sync(0xffffffffu, n > 0)), big = __reduce_add_sync(0xffffffffu, nb),
                 bigrows = __reduce_add_sync(0xffffffffu, tensor ? n : 0), tall = __popc(__ballot_sync(0xffffffffu, len > few));
  if (in) {
    for (uint32_t i = lane; i < kTileN / 2; i += 32) ((uint32_t *)s_len[warp])[i] = 0;
    if (lane == 31) s_sum[0][warp] = v[0], s_sum[1][warp] = v[1], s_sum[2][warp] = v[2], s_sum[3][warp] = v[3];
    if (lane == 0) s_sum[4][warp] = hit, s_sum[5][warp] = big, s_sum[6][warp] = bigrows, s_sum[7][warp] = tall;
    __syncwarp();
  }
  const uint32_t same = __match_any_sync(0xffffffffu, len);
  if (in && len && (uint32_t)__ffs(same) - 1 == lane) s_len[warp][len] = (uint16_t)__popc(same);
  __syncthreads();
  // Thread e < 256 has the tiles of length e: how many come before each warp's, and (below) before all of that length.
  uint32_t longer = 0;
  if (e < kTileN) {
    uint32_t sum = 0;
#pragma unroll
    for (uint32_t w = 0; w < kWarps; w++) {
      const uint32_t c = s_len[w][e];
      s_len[w][e] = (uint16_t)sum;
      sum += c;
    }
    longer = sum;
#pragma unroll
    for (uint32_t off = 1; off < 32; off <<= 1) {
      const uint32_t u = __shfl_down_sync(0xffffffffu, longer, off);
      if (lane + off < 32) longer += u;
    }
    if (lane == 0) s_bin[warp] = longer;
    longer -= sum;  // within the warp's 32 lengths
  }
  __syncthreads();
  if (e < kTileN) {
    for (uint32_t w = warp + 1; w < kTileN / 32; w++) longer += s_bin[w];
#pragma unroll
    for (uint32_t w = 0; w < kWarps; w++) s_len[w][e] = (uint16_t)(s_len[w][e] + longer);
  }
  __syncthreads();
  uint32_t all[kSums], before[4];
#pragma unroll
  for (int j = 0; j < (int)kSums; j++) {
    const uint32_t b = before_and_all(s_sum[j], all[j]);
    if (j < 4) before[j] = b + v[j];
  }
  const uint32_t first = in ? before[0] - n : 0;
  if (e < NE) {
    o.cnt[e] = n;
    o.base[e] = first;
    const uint32_t tile0 = before[1] - nt, group0 = before[2] - ng, big0 = before[3] - mine;
    for (uint32_t i = 0; i < nt; i++)
      o.tiles[tile0 + i] = MoeTile{first_expert + e, e, first + i * kTileRows, min(kTileRows, n - i * kTileRows)};
    for (uint32_t i = 0; i < ng; i++)
      o.groups[group0 + i] = MoeGroup{e, first + i * group_max, min(group_max, n - i * group_max)};
    for (uint32_t i = 0; i < mine; i++) o.big[big0 + i] = BigTile{e, first + i * kTileN, i < nfull ? kTileN : rem};
    if (len) o.big[all[3] + s_len[warp][len] + __popc(same & ((1u << lane) - 1))] = BigTile{e, first, rem};
  }
  if (e == 511) {
    o.counters[0] = all[1], o.counters[1] = all[2], o.counters[2] = all[4], o.counters[3] = all[0];
    o.counters[4] = all[5], o.counters[5] = all[6], o.counters[6] = all[3] + all[7];
  }
  return first;
}

// The scan over a long step's chunks in two levels: a CTA per kScanGroup chunks leaves every expert's running count
// within its group in chunk_off and the group's total in group_tot; k_pack_scan then walks the groups' totals instead
// of the chunks, and k_pack_fill adds a chunk's group's offset to the chunk's own. (One CTA walking a thousand chunks
// took 133 us of a 32,768-row step.)
constexpr uint32_t kScanGroup = 32;
static __global__ void __launch_bounds__(512) k_pack_scan_groups(const uint32_t *chunk_hist, uint32_t nchunks, uint32_t NE,
                                                         uint32_t *__restrict__ chunk_off, uint32_t *__restrict__ group_tot) {
  dependents_may_launch(), wait_for_predecessors();
  const uint32_t e = threadIdx.x, c_begin = blockIdx.x * kScanGroup, c_end = min(nchunks, c_begin + kScanGroup);
  if (e >= NE) return;
  uint32_t run = 0;
  for (uint32_t c0 = c_begin; c0 < c_end; c0 += 16) {
    uint32_t v[16];
#pragma unroll
    for (uint32_t j = 0; j < 16; j++) v[j] = c0 + j < c_end ? chunk_hist[(uint64_t)(c0 + j) * NE + e] : 0;
#pragma unroll
    for (uint32_t j = 0; j < 16; j++) {
      if (c0 + j < c_end) chunk_off[(uint64_t)(c0 + j) * NE + e] = run;
      run += v[j];
    }
  }
  group_tot[(uint64_t)blockIdx.x * NE + e] = run;
}

// groups: null, or the groups' totals left by k_pack_scan_groups, [ngroups][NE], which become the groups' offsets in place.
static __global__ void __launch_bounds__(512) k_pack_scan(const uint32_t *chunk_hist, uint32_t nchunks, uint32_t NE,
                                                  uint32_t first_expert, uint32_t tensor_min, uint32_t tensor_budget, uint32_t group_max,
                                                  PackOut o, uint32_t *__restrict__ groups = nullptr, uint32_t ngroups = 0) {
  dependents_may_launch(), wait_for_predecessors();
  const uint32_t e = threadIdx.x;
  uint32_t run = 0;
  if (e < NE && groups) {
    for (uint32_t g0 = 0; g0 < ngroups; g0 += 16) {
      uint32_t v[16];
#pragma unroll
      for (uint32_t j = 0; j < 16; j++) v[j] = g0 + j < ngroups ? groups[(uint64_t)(g0 + j) * NE + e] : 0;
#pragma unroll
      for (uint32_t j = 0; j < 16; j++) {
        if (g0 + j < ngroups) groups[(uint64_t)(g0 + j) * NE + e] = run;
        run += v[j];
      }
    }
  } else if (e < NE) {
    // Sixteen chunks' counts are loaded at once: a lone CTA walking a thousand chunks one load at a time would spend
    // the stage on memory latency.
    for (uint32_t c0 = 0; c0 < nchunks; c0 += 16) {
      uint32_t v[16];
#pragma unroll
      for (uint32_t j = 0; j < 16; j++) v[j] = c0 + j < nchunks ? chunk_hist[(uint64_t)(c0 + j) * NE + e] : 0;
#pragma unroll
      for (uint32_t j = 0; j < 16; j++) {
        if (c0 + j < nchunks) o.chunk_off[(uint64_t)(c0 + j) * NE + e] = run;
        run += v[j];
      }
    }
  }
  pack_scan_block(e, run, NE, first_expert, tensor_min, tensor_budget, group_max, o);
}

// One CTA per chunk: the chunk's entries take their expert's rows in the order they stand in.
// inv[a] = row; row_src[row] = a / src_div (the activation row the assignment reads: its token). Dynamic shared
// memory 16 * NE words.
static __global__ void __launch_bounds__(512) k_pack_fill(const int32_t *ids, uint32_t A, uint32_t chunk_len, uint32_t NE,
                                                  const uint32_t *base, const uint32_t *chunk_off,
                                                  uint32_t src_div, uint32_t *__restrict__ inv, uint32_t *__restrict__ row_src,
                                                  uint32_t first_expert = 0, const uint32_t *group_off = nullptr) {
  dependents_may_launch(), wait_for_predecessors();
  // A thread an entry (chunk_len <= 512). An entry's row is its expert's first row for this chunk plus the number of
  // the chunk's earlier entries with the same expert: those of earlier warps, counted per (warp, expert) in shared
  // memory and summed over the warps, and those of lower lanes of its own warp, which match_any names. (A thread an
  // expert, each walking the chunk's entries, took 52 us of a 32,768-row step.)
  extern __shared__ uint32_t s_cnt[];  // [16][NE]
  const uint32_t a0 = blockIdx.x * chunk_len, n = min(A, a0 + chunk_len) - a0;
  const uint32_t i = threadIdx.x, warp = i / 32, lane = i % 32;
  for (uint32_t k = i; k < 16 * NE; k += 512) s_cnt[k] = 0;
  const uint32_t e = i < n ? (uint32_t)ids[a0 + i] - first_expert : 0xFFFFFFFFu;
  const bool valid = e < NE;
  // Entries with no expert here get a key of their own, so that they match nothing.
  const uint32_t same = __match_any_sync(0xffffffffu, valid ? e : NE + lane);
  const uint32_t before = __popc(same & ((1u << lane) - 1));
  __syncthreads();
  if (valid && before == 0) s_cnt[warp * NE + e] = __popc(same);
  __syncthreads();
  if (i < NE) {
    uint32_t run = 0;
    for (uint32_t w = 0; w < 16; w++) {
      const uint32_t c = s_cnt[w * NE + i];
      s_cnt[w * NE + i] = run;
      run += c;
    }
  }
  __syncthreads();
  if (!valid) return;
  uint32_t row = base[e] + chunk_off[(uint64_t)blockIdx.x * NE + e] + s_cnt[warp * NE + e] + before;
  if (group_off) row += group_off[(uint64_t)(blockIdx.x / kScanGroup) * NE + e];
  inv[a0 + i] = row;
  row_src[row] = (a0 + i) / src_div;
}

// A step of a few rows (one chunk of the pack at most, kChunkTokens rows): top-k, scan and fill in one CTA, four launches
// less for the steps that launches bound. Dynamic shared memory kChunkTokens * K words for the chunk's ids.
static __global__ void __launch_bounds__(32 * kChunkTokens, 1) k_router_topk_pack(const float *rl, const float *__restrict__ bias, uint32_t T,
                                                                       uint32_t NE, uint32_t K, int32_t *__restrict__ ids, float *__restrict__ w,
                                                                       float *__restrict__ gs, uint32_t tensor_min, uint32_t tensor_budget,
                                                                       uint32_t group_max, PackOut o, uint32_t *__restrict__ inv,
                                                                       uint32_t *__restrict__ row_src) {
  __shared__ uint32_t hist[512];
  extern __shared__ int32_t s_chunk_ids[];
  dependents_may_launch(), wait_for_predecessors();
  router_topk_block(rl, RouterApprox{}, bias, T, NE, K, ids, w, gs, hist, s_chunk_ids);
  const uint32_t e = threadIdx.x;
  const uint32_t run = e < NE ? hist[e] : 0;
  uint32_t row = pack_scan_block(e, run, NE, 0, tensor_min, tensor_budget, group_max, o);
  if (e < NE && run) {
    const uint32_t A = T * K;
    for (uint32_t i = 0; i < A; i++)
      if ((uint32_t)s_chunk_ids[i] == e) {
        inv[i] = row;
        row_src[row] = i / K;
        row++;
      }
  }
}

// A short step's route by one CTA: the top-k of at most kShortRows rows, a warp each, and its lists.
static __global__ void __launch_bounds__(32 * kShortRows) k_short_route(const ShortRoute rt) {
  __shared__ uint32_t s_ids[kShortMax];
  dependents_may_launch(), wait_for_predecessors();
  short_route(rt, s_ids, true);
}

// ---------------------------------------------------------------------------------------------------------------
// Combine: out[t] = sum over k, in rank order, of w[t][k] * y[inv[t K + k]] + gs[t] * s[t], in f32 (layer.cl:874-877).
// One CTA per row. y is f32, or f16 when the tile kernels or other GPUs left it in that form. With res set, the row's
// residual res[t] is added last: a stack's x <- x + block(x) without a kernel of its own.
__device__ __forceinline__ float4 load_row4(const float *y, uint64_t row, uint32_t E, uint32_t i) { return ((const float4 *)(y + row * E))[i]; }
__device__ __forceinline__ float4 load_row4(const __half *y, uint64_t row, uint32_t E, uint32_t i) {
  const uint2 u = ((const uint2 *)(y + row * E))[i];
  const float2 a = __half22float2(*(const __half2 *)&u.x), b = __half22float2(*(const __half2 *)&u.y);
  return make_float4(a.x, a.y, b.x, b.y);
}
template <class Y>
static __global__ void __launch_bounds__(256) k_combine(const Y *y, const uint32_t *inv, const float *w, const float *gs, const float *s, uint32_t K,
                                                       uint32_t E, float *out, const float *res) {
  dependents_may_launch(), wait_for_predecessors();
  const uint32_t t = blockIdx.x;
  __shared__ uint32_t rows[16];
  __shared__ float wk[16];
  if (threadIdx.x < K) rows[threadIdx.x] = inv[(uint64_t)t * K + threadIdx.x], wk[threadIdx.x] = w[(uint64_t)t * K + threadIdx.x];
  __syncthreads();
  const float g = s ? gs[t] : 0.0f;
  for (uint32_t i = threadIdx.x; i < E / 4; i += 256) {
    float4 acc = make_float4(0, 0, 0, 0);
    for (uint32_t k = 0; k < K; k++) {
      const float4 v = load_row4(y, rows[k], E, i);
      acc.x = fmaf(wk[k], v.x, acc.x), acc.y = fmaf(wk[k], v.y, acc.y);
      acc.z = fmaf(wk[k], v.z, acc.z), acc.w = fmaf(wk[k], v.w, acc.w);
    }
    if (s) {
      const float4 v = ((const float4 *)(s + (uint64_t)t * E))[i];
      acc.x = fmaf(g, v.x, acc.x), acc.y = fmaf(g, v.y, acc.y), acc.z = fmaf(g, v.z, acc.z), acc.w = fmaf(g, v.w, acc.w);
    }
    if (res) {
      const float4 v = ((const float4 *)(res + (uint64_t)t * E))[i];
      acc.x += v.x, acc.y += v.y, acc.z += v.z, acc.w += v.w;
    }
    ((float4 *)(out + (uint64_t)t * E))[i] = acc;
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Expert parallel: the rows that cross GPUs. A wire row is one quantised activation row packed: K codes, its scales,
// q8_K's sums, padded to 16 bytes.
__host__ __device__ constexpr uint32_t wire_row_bytes(bool q8k, uint32_t K) { return (K + (q8k ? K / 64 + K / 8 : K / 8) + 15) & ~15u; }

// wire[r] = the quantised row of the token assignment row r reads (row_src[r]); ids_sorted[r] = its expert. One warp
// per row.
static __global__ void __launch_bounds__(256) k_gather_wire(const ActView act, uint32_t K, bool q8k, const uint32_t *__restrict__ row_src,
                                                           const uint32_t *__restrict__ inv, const int32_t *__restrict__ ids, uint32_t A,
                                                           uint8_t *__restrict__ wire, int32_t *__restrict__ ids_sorted) {
  const uint32_t lane = threadIdx.x % 32;
  const uint64_t r = (uint64_t)blockIdx.x * 8 + threadIdx.x / 32;
  if (r >= A) return;
  const uint32_t wb = wire_row_bytes(q8k, K), t = row_src[r], dbytes = q8k ? K / 64 : K / 8;
  uint8_t *dst = wire + r * wb;
  const int4 *q = (const int4 *)(act.q + (uint64_t)t * act.q_stride);
  for (uint32_t i = lane; i < K / 16; i += 32) ((int4 *)dst)[i] = q[i];
  const uint32_t *d = (const uint32_t *)((const uint8_t *)act.d + (uint64_t)t * act.d_stride);
  for (uint32_t i = lane; i < dbytes / 4; i += 32) ((uint32_t *)(dst + K))[i] = d[i];
  if (q8k) {
    const uint32_t *b = (const uint32_t *)((const uint8_t *)act.bs + (uint64_t)t * act.bs_stride);
    for (uint32_t i = lane; i < K / 32; i += 32) ((uint32_t *)(dst + K + dbytes))[i] = b[i];
  }
  // The ids in expert order: assignment a sits at row inv[a]. Here r also counts the assignments.
  if (lane == 0) ids_sorted[inv[r]] = ids[r];
}

// The f16 operand of the tensor-core kernels from wire rows: code * scale, as the quantisers write it. One warp per
// 256 values. row_stride: bytes from a row to the next when they carry more than the row itself (0: none).
// With place_of, a row goes straight to its places in expert order instead of to its own index: row r has up to
// `places` entries, entry k with an expert when ids[r * places + k] >= 0 and then at row place_of[r * places + k] of
// out's out_rows rows.
static __global__ void __launch_bounds__(256) k_wire_to_f16(const uint8_t *__restrict__ wire, uint32_t K, bool q8k, uint64_t nblk256,
                                                           __half *__restrict__ out, uint32_t row_stride = 0,
                                                           const int32_t *__restrict__ ids = nullptr, const uint32_t *__restrict__ place_of = nullptr,
                                                           uint32_t places = 0, uint64_t out_rows = 0) {
  const uint64_t blk = (uint64_t)blockIdx.x * 8 + threadIdx.x / 32;
  if (blk >= nblk256) return;
  const uint32_t lane = threadIdx.x % 32, per_row = K / 256, wb = row_stride ? row_stride : wire_row_bytes(q8k, K);
  const uint64_t row = blk / per_row;
  const uint32_t b = (uint32_t)(blk % per_row);
  const uint8_t *src = wire + row * wb;
  const char4 lo = ((const char4 *)(src + 256 * b))[2 * lane], hi = ((const char4 *)(src + 256 * b))[2 * lane + 1];
  const float d = q8k ? ((const float *)(src + K))[b] : ((const float *)(src + K))[8 * b + lane / 4];
  const __half2 h0 = __floats2half2_rn(d * (float)lo.x, d * (float)lo.y), h1 = __floats2half2_rn(d * (float)lo.z, d * (float)lo.w);
  const __half2 h2 = __floats2half2_rn(d * (float)hi.x, d * (float)hi.y), h3 = __floats2half2_rn(d * (float)hi.z, d * (float)hi.w);
  uint4 o;
  o.x = *(const uint32_t *)&h0, o.y = *(const uint32_t *)&h1, o.z = *(const uint32_t *)&h2, o.w = *(const uint32_t *)&h3;
  if (!place_of) {
    ((uint4 *)(out + row * K + 256 * b))[lane] = o;
    return;
  }
  // A place past out's rows can only come from an id that is not one of this GPU's experts (the pack leaves such an
  // entry's place unset): it is skipped, not written.
  for (uint32_t k = 0; k < places; k++) {
    if (__ldg(ids + row * places + k) < 0) continue;
    const uint64_t place = __ldg(place_of + row * places + k);
    if (place < out_rows) ((uint4 *)(out + place * K + 256 * b))[lane] = o;
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Expert parallel with one row per (token, GPU). A token's K experts live on a few GPUs (about 5.9 of 8, 2.0 of 2 for
// K = 10 and even routing), so a token's quantised row travels once to each GPU that holds any of its experts, with the
// list of those experts and their routing weights beside it; the GPU returns one row, the weighted sum of its experts'
// results for the token. GPUs own contiguous ranges of `per` experts.
constexpr uint32_t kMaxWorld = 8;
constexpr uint32_t kDestChunk = 256;                   // tokens a CTA plans
constexpr uint32_t kMetaBytes = 2 * 16 + 4 * 16;       // a travelling row's list: 16 u16 local expert ids, 16 f32 weights
__host__ __device__ constexpr uint32_t dispatch_row_bytes(bool q8k, uint32_t K) { return wire_row_bytes(q8k, K) + kMetaBytes; }

// Per chunk of tokens: how many of them go to each GPU, and how many assignments go with them.
static __global__ void __launch_bounds__(kDestChunk) k_dest_count(const int32_t *__restrict__ ids, uint32_t T, uint32_t K, uint32_t per,
                                                                uint32_t *__restrict__ chunk_cnt, uint32_t *__restrict__ chunk_asg) {
  __shared__ uint32_t rows[kMaxWorld], asg[kMaxWorld];
  if (threadIdx.x < kMaxWorld) rows[threadIdx.x] = 0, asg[threadIdx.x] = 0;
  __syncthreads();
  const uint32_t t = blockIdx.x * kDestChunk + threadIdx.x;
  if (t < T) {
    uint32_t mask = 0;
    for (uint32_t k = 0; k < K; k++) {
      const uint32_t g = (uint32_t)ids[(uint64_t)t * K + k] / per;
      atomicAdd(&asg[g], 1u);
      mask |= 1u << g;
    }
    for (uint32_t g = 0; g < kMaxWorld; g++)
      if (mask >> g & 1) atomicAdd(&rows[g], 1u);
  }
  __syncthreads();
  if (threadIdx.x < kMaxWorld) {
    chunk_cnt[blockIdx.x * kMaxWorld + threadIdx.x] = rows[threadIdx.x];
    chunk_asg[blockIdx.x * kMaxWorld + threadIdx.x] = asg[threadIdx.x];
  }
}

// pos[t][g] = the place of token t's row among those this GPU sends to GPU g, in token order, or 0xFFFFFFFF when none
// of its experts lives there. totals[g] = rows for GPU g, totals[kMaxWorld + g] = assignments for it (written by CTA 0).
static __global__ void __launch_bounds__(kDestChunk) k_dest_fill(const int32_t *__restrict__ ids, uint32_t T, uint32_t K, uint32_t per,
                                                               const uint32_t *__restrict__ chunk_cnt, const uint32_t *__restrict__ chunk_asg,
                                                               uint32_t nchunks, uint32_t *__restrict__ pos, uint32_t *__restrict__ totals) {
  __shared__ uint32_t base[kMaxWorld], warp_cnt[kDestChunk / 32][kMaxWorld], tot[2 * kMaxWorld];
  if (threadIdx.x < kMaxWorld) base[threadIdx.x] = 0;
  if (threadIdx.x < 2 * kMaxWorld) tot[threadIdx.x] = 0;
  __syncthreads();
  // The chunks before this one (and, for CTA 0, all of them for the totals).
  for (uint32_t i = threadIdx.x; i < nchunks * kMaxWorld; i += kDestChunk) {
    const uint32_t c = i / kMaxWorld, g = i % kMaxWorld;
    if (c < blockIdx.x && chunk_cnt[i]) atomicAdd(&base[g], chunk_cnt[i]);
    if (blockIdx.x == 0) atomicAdd(&tot[g], chunk_cnt[i]), atomicAdd(&tot[kMaxWorld + g], chunk_asg[i]);
  }
  const uint32_t t = blockIdx.x * kDestChunk + threadIdx.x, lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  uint32_t mask = 0;
  if (t < T)
    for (uint32_t k = 0; k < K; k++) mask |= 1u << ((uint32_t)ids[(uint64_t)t * K + k] / per);
  uint32_t rank[kMaxWorld];
#pragma unroll
  for (uint32_t g = 0; g < kMaxWorld; g++) {
    const uint32_t b = __ballot_sync(0xffffffffu, mask >> g & 1);
    rank[g] = __popc(b & ((1u << lane) - 1));
    if (lane == 0) warp_cnt[warp][g] = __popc(b);
  }
  __syncthreads();
  if (t < T) {
#pragma unroll
    for (uint32_t g = 0; g < kMaxWorld; g++) {
      uint32_t before = base[g];
      for (uint32_t w = 0; w < warp; w++) before += warp_cnt[w][g];
      pos[(uint64_t)t * kMaxWorld + g] = (mask >> g & 1) ? before + rank[g] : 0xFFFFFFFFu;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x < 2 * kMaxWorld) totals[threadIdx.x] = tot[threadIdx.x];
}

// The travelling rows, destination by destination (GPU 0's first), each destination's in token order: the token's
// quantised row as k_gather_wire lays it, then its experts on that GPU as local indices (0xFFFF: none) in rank order,
// then their routing weights. One warp per (token, GPU).
static __global__ void __launch_bounds__(256) k_dispatch_rows(const ActView act, uint32_t E, bool q8k, const int32_t *__restrict__ ids,
                                                             const float *__restrict__ w, const uint32_t *__restrict__ pos,
                                                             const uint32_t *__restrict__ totals, uint32_t T, uint32_t K, uint32_t per,
                                                             uint32_t world, uint8_t *__restrict__ out) {
  const uint32_t lane = threadIdx.x % 32;
  const uint64_t pair = (uint64_t)blockIdx.x * 8 + threadIdx.x / 32;
  if (pair >= (uint64_t)T * world) return;
  const uint32_t t = (uint32_t)(pair / world), g = (uint32_t)(pair % world), p = pos[(uint64_t)t * kMaxWorld + g];
  if (p == 0xFFFFFFFFu) return;
  uint32_t first = 0;
  for (uint32_t i = 0; i < g; i++) first += totals[i];
  const uint32_t wb = wire_row_bytes(q8k, E), dbytes = q8k ? E / 64 : E / 8;
  uint8_t *dst = out + (uint64_t)(first + p) * (wb + kMetaBytes);
  const int4 *q = (const int4 *)(act.q + (uint64_t)t * act.q_stride);
  for (uint32_t i = lane; i < E / 16; i += 32) ((int4 *)dst)[i] = q[i];
  const uint32_t *d = (const uint32_t *)((const uint8_t *)act.d + (uint64_t)t * act.d_stride);
  for (uint32_t i = lane; i < dbytes / 4; i += 32) ((uint32_t *)(dst + E))[i] = d[i];
  if (q8k) {
    const uint32_t *b = (const uint32_t *)((const uint8_t *)act.bs + (uint64_t)t * act.bs_stride);
    for (uint32_t i = lane; i < E / 32; i += 32) ((uint32_t *)(dst + E + dbytes))[i] = b[i];
  }
  if (lane < 16) {
    uint32_t local = 0xFFFFu;
    float wk = 0.0f;
    if (lane < K) {
      const uint32_t e = (uint32_t)ids[(uint64_t)t * K + lane];
      if (e / per == g) local = e % per, wk = w[(uint64_t)t * K + lane];
    }
    ((uint16_t *)(dst + wb))[lane] = (uint16_t)local;
    ((float *)(dst + wb + 32))[lane] = wk;
  }
}

// The lists of the rows received, flattened: ids[r * K + k] = first_expert + the local index, or -1 for no expert;
// w[r * K + k] its weight. One thread per entry.
static __global__ void __launch_bounds__(256) k_meta_unpack(const uint8_t *__restrict__ rows, uint64_t R, uint32_t wb, uint32_t K,
                                                           uint32_t first_expert, int32_t *__restrict__ ids, float *__restrict__ w) {
  const uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= R * K) return;
  const uint8_t *meta = rows + (i / K) * (wb + kMetaBytes) + wb;
  const uint32_t local = ((const uint16_t *)meta)[i % K];
  ids[i] = local == 0xFFFFu ? -1 : (int32_t)(first_expert + local);
  w[i] = ((const float *)(meta + 32))[i % K];
}

// What a GPU returns for a received row: the weighted sum of its experts' results for the row, in the row's rank
// order, f32 accumulate, as f16. One CTA per row.
template <class Y>
static __global__ void __launch_bounds__(256) k_combine_partial(const Y *__restrict__ y, const uint32_t *__restrict__ inv,
                                                               const int32_t *__restrict__ ids, const float *__restrict__ w, uint32_t K,
                                                               uint32_t E, __half *__restrict__ out) {
  const uint64_t r = blockIdx.x;
  __shared__ uint32_t rows[16];
  __shared__ float wk[16];
  __shared__ uint32_t n;
  if (threadIdx.x == 0) {
    uint32_t m = 0;
    for (uint32_t k = 0; k < K; k++)
      if (ids[r * K + k] >= 0) rows[m] = inv[r * K + k], wk[m] = w[r * K + k], m++;
    n = m;
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < E / 4; i += 256) {
    float4 acc = make_float4(0, 0, 0, 0);
    for (uint32_t k = 0; k < n; k++) {
      const float4 v = load_row4(y, rows[k], E, i);
      acc.x = fmaf(wk[k], v.x, acc.x), acc.y = fmaf(wk[k], v.y, acc.y);
      acc.z = fmaf(wk[k], v.z, acc.z), acc.w = fmaf(wk[k], v.w, acc.w);
    }
    const __half2 a = __floats2half2_rn(acc.x, acc.y), b = __floats2half2_rn(acc.z, acc.w);
    uint2 o;
    o.x = *(const uint32_t *)&a, o.y = *(const uint32_t *)&b;
    ((uint2 *)(out + r * E))[i] = o;
  }
}

// At home: out[t] = the GPUs' partial sums for token t added in GPU order, + gs[t] * s[t] (+ res[t]). back holds the
// rows as they were sent: destination by destination. One CTA per token.
static __global__ void __launch_bounds__(256) k_combine_home(const __half *__restrict__ back, const uint32_t *__restrict__ pos,
                                                            const uint32_t *__restrict__ totals, const float *__restrict__ gs,
                                                            const float *__restrict__ s, const float *__restrict__ res, uint32_t world,
                                                            uint32_t E, float *__restrict__ out) {
  const uint32_t t = blockIdx.x;
  __shared__ uint32_t rows[kMaxWorld];
  __shared__ uint32_t n;
  if (threadIdx.x == 0) {
    uint32_t m = 0, first = 0;
    for (uint32_t g = 0; g < world; g++) {
      const uint32_t p = pos[(uint64_t)t * kMaxWorld + g];
      if (p != 0xFFFFFFFFu) rows[m++] = first + p;
      first += totals[g];
    }
    n = m;
  }
  __syncthreads();
  const float g = s ? gs[t] : 0.0f;
  for (uint32_t i = threadIdx.x; i < E / 4; i += 256) {
    float4 acc = make_float4(0, 0, 0, 0);
    for (uint32_t k = 0; k < n; k++) {
      const float4 v = load_row4(back, rows[k], E, i);
      acc.x += v.x, acc.y += v.y, acc.z += v.z, acc.w += v.w;
    }
    if (s) {
      const float4 v = ((const float4 *)(s + (uint64_t)t * E))[i];
      acc.x = fmaf(g, v.x, acc.x), acc.y = fmaf(g, v.y, acc.y), acc.z = fmaf(g, v.z, acc.z), acc.w = fmaf(g, v.w, acc.w);
    }
    if (res) {
      const float4 v = ((const float4 *)(res + (uint64_t)t * E))[i];
      acc.x += v.x, acc.y += v.y, acc.z += v.z, acc.w += v.w;
    }
    ((float4 *)(out + (uint64_t)t * E))[i] = acc;
  }
}

// out[r] = y[inv[r]]: the experts' rows back in the order they arrived, f32 or f16 on either side. One CTA per row.
template <class Y, class O>
static __global__ void __launch_bounds__(256) k_unpermute(const Y *__restrict__ y, const uint32_t *__restrict__ inv, uint32_t E,
                                                         O *__restrict__ out) {
  const uint64_t r = blockIdx.x, src = inv[r];
  for (uint32_t i = threadIdx.x; i < E / 4; i += 256) {
    if constexpr (sizeof(Y) == 2 && sizeof(O) == 2) {
      ((uint2 *)(out + r * E))[i] = ((const uint2 *)(y + src * E))[i];
    } else {
      const float4 v = load_row4(y, src, E, i);
      if constexpr (sizeof(O) == 4) {
        ((float4 *)(out + r * E))[i] = v;
      } else {
        const __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
        uint2 o;
        o.x = *(const uint32_t *)&a, o.y = *(const uint32_t *)&b;
        ((uint2 *)(out + r * E))[i] = o;
      }
    }
  }
}

}  // namespace moe

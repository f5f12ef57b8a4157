// The router's top-k: a row's experts, their renormalised weights and the shared expert's gate from its logits, exact or
// approximate, by one warp. (The reference's router / p_router: kernels/models/qwen4exp/layer.cl:765-847,
// prompt.cl:652-678, route.h:39-98.)
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace moe {

constexpr uint32_t kRouterPieces = 8;   // pieces a router product is summed in

// ---------------------------------------------------------------------------------------------------------------
// Top-k. One warp per row, lane holding experts lane + 32 j. Keys order the logits as floats do (the reference's
// topk_key, kernels/include/topk.h:12-15), -0 taken as +0; winners come out largest first, ties to the lower expert
// (route.h:33-38). Weights: p_k = exp(v_k - max) / sum, w_k = p_k / max(sum of the K p's, 6.1035e-5)
// (layer.cl:784-787). The CTA's rows are one chunk of the pack: it leaves the chunk's count of every expert.
__device__ __forceinline__ uint32_t order_key(float v) {
  const uint32_t u = __float_as_uint(v + 0.0f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
}

constexpr int kMaxPerLane = 16;  // experts a lane holds at most: 512 / 32

// Steps of many rows: the logits come from the tensor-core product (router_mma.cuh) and are approximate. For row t
// every one is within eps_t of the logit the exact order gives, eps_t = eps_rel * |x_t| + eps_abs (setup_router_tensor),
// with |x_t|^2 summed from norm2_parts. The top-k below then recomputes, in the exact order, only what that bound
// cannot decide.
struct RouterApprox {
  float *logits;             // [parts][T][NE], to be added up (the sum is left in part 0); null: the logits are exact rows rl[t][NE + 1]
  const float *x;            // [T][E]
  const float *W;            // [NE][E]
  const float *norm2_parts;  // [T][nparts]
  const float *gate_parts;   // [T][nparts]: the parts of the shared expert's gate logit
  uint32_t E, nparts;
  uint32_t parts;
  uint64_t part_stride;      // T * NE
  float eps_rel, eps_abs;
};

// The logits of up to four experts for row x, each exactly as k_router_logits_rows and the CPU oracle sum it: eight
// pieces of the row, each a chain of fused multiply-adds from 0 in index order, the pieces added in order, the bias
// last. Lane 8 j + s takes piece s of expert ex[j]; lanes 8 j .. 8 j + 7 return expert ex[j]'s logit.
__device__ __forceinline__ float exact_logits4(const float *x, const float *__restrict__ W, const float *__restrict__ bias,
                                               uint32_t E, uint32_t e, uint32_t lane) {
  const uint32_t piece = E / kRouterPieces, s = lane % 8;
  const float4 *xp = (const float4 *)(x + s * piece), *wp = (const float4 *)(W + (uint64_t)e * E + s * piece);
  float p = 0.0f;
  // Eight loads of each operand in flight a lane: the chain of multiply-adds is short beside a trip to memory, so the
  // pass costs about piece / 32 such trips.
  for (uint32_t i = 0; i < piece / 4; i += 8) {
    float4 xv[8], wv[8];
#pragma unroll
    for (int j = 0; j < 8; j++) xv[j] = xp[i + j], wv[j] = __ldg(wp + i + j);
#pragma unroll
    for (int j = 0; j < 8; j++) {
      p = fmaf(xv[j].x, wv[j].x, p);
      p = fmaf(xv[j].y, wv[j].y, p);
      p = fmaf(xv[j].z, wv[j].z, p);
      p = fmaf(xv[j].w, wv[j].w, p);
    }
  }
  float tot = __shfl_sync(0xffffffffu, p, lane & ~7u);
#pragma unroll
  for (int j = 1; j < (int)kRouterPieces; j++) tot = __fadd_rn(tot, __shfl_sync(0xffffffffu, p, (lane & ~7u) + j));
  if (bias) tot = __fadd_rn(tot, bias[e]);
  return tot;
}

// exact_logits4 with the operands brought through shared memory. A lane walking its own piece of a row from global
// memory touches, with the other lanes, 32 different lines an instruction, and the tag stage of L1 then sets the pace
// (measured: two thirds of its peak, the kernel's limit). Here the warp copies the row and the four experts' rows
// chunk by chunk with 16-byte asynchronous copies, eight lanes to a piece's 128 contiguous bytes, the next chunk on
// its way while this one is summed; the lanes read their pieces from shared memory, whose padding (a piece's chunk
// every 144 bytes) spreads a quarter-warp's eight 16-byte reads over all banks. The sums are the same chains.
constexpr uint32_t kExChunk = 32;                        // values of each piece a chunk holds
constexpr uint32_t kExPiece = kExChunk * 4 + 16;         // bytes from one piece's chunk to the next in shared memory
constexpr uint32_t kExRow = kRouterPieces * kExPiece;    // a row's chunk: 1,152 bytes
constexpr uint32_t kExBuf = 5 * kExRow;                  // the row and four experts' rows
constexpr uint32_t kExWarpBytes = 2 * kExBuf;            // two chunks: 11,520 bytes a warp
__device__ __forceinline__ void cp_async16(uint32_t dst_smem, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src) : "memory");
}
// With fewer than four experts (n) only their rows are copied; the other lanes' sums are nobody's.
__device__ __forceinline__ float exact_logits4_staged(const float *x, const float *__restrict__ W, const float *__restrict__ bias,
                                                      uint32_t E, uint32_t e, uint32_t n, uint32_t lane, uint8_t *buf) {
  const uint32_t piece = E / kRouterPieces, nch = piece / kExChunk, s = lane % 8, g = lane / 8;
  const uint32_t buf32 = (uint32_t)__cvta_generic_to_shared(buf);
  // The four experts of the pass, known to every lane.
  uint32_t ex[4];
#pragma unroll
  for (int j = 0; j < 4; j++) ex[j] = __shfl_sync(0xffffffffu, e, 8 * j);
  auto issue = [&](uint32_t c, uint32_t b) {
    // A row's chunk is 8 pieces x 128 bytes: 64 copies of 16 bytes, two a lane.
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const uint32_t idx = k * 32 + lane, pc = idx / 8, j = idx % 8;
      const uint64_t off = (uint64_t)pc * piece + c * kExChunk + j * 4;
      const uint32_t dst = buf32 + b * kExBuf + pc * kExPiece + j * 16;
      cp_async16(dst, x + off);
#pragma unroll
      for (int r = 0; r < 4; r++)
        if ((uint32_t)r < n) cp_async16(dst + (1 + r) * kExRow, W + (uint64_t)ex[r] * E + off);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float p = 0.0f;
  issue(0, 0);
  for (uint32_t c = 0; c < nch; c++) {
    if (c + 1 < nch) {
      issue(c + 1, (c + 1) & 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncwarp();
    const float4 *xs = (const float4 *)(buf + (c & 1) * kExBuf + s * kExPiece);
    const float4 *ws = (const float4 *)(buf + (c & 1) * kExBuf + (1 + g) * kExRow + s * kExPiece);
#pragma unroll
    for (int j = 0; j < (int)kExChunk / 4; j++) {
      const float4 xv = xs[j], wv = ws[j];
      p = fmaf(xv.x, wv.x, p);
      p = fmaf(xv.y, wv.y, p);
      p = fmaf(xv.z, wv.z, p);
      p = fmaf(xv.w, wv.w, p);
    }
    __syncwarp();  // every lane has read the chunk before its buffer is filled again
  }
  float tot = __shfl_sync(0xffffffffu, p, lane & ~7u);
#pragma unroll
  for (int j = 1; j < (int)kRouterPieces; j++) tot = __fadd_rn(tot, __shfl_sync(0xffffffffu, p, (lane & ~7u) + j));
  if (bias) tot = __fadd_rn(tot, bias[e]);
  return tot;
}

// Row t's part, by a warp: its ids, weights and gate written, its experts counted in hist (shared, 512 words) and put in
// s_ids (shared, K words), each where not null. With w null (exact logits only) nothing but s_ids is written, and the
// softmax, which only the weights need, is left out. ex_buf: kExWarpBytes of shared memory of the warp's own, through which
// the exact sums then take their operands (E a multiple of 8 * kExChunk); null: straight from global memory.
//
// With approximate logits a row's candidates are the experts whose approximate logit is within 2 eps of the K-th
// largest: the true top K is among them (an expert outside is below K others by more than the two errors can
// bridge). Sorted by approximate logit, two neighbours less than 2 eps apart cannot be ordered by it, and both get
// their exact logit; any other pair's order is certain. The candidates are then ranked by (logit, lower expert first)
// with exact logits where they were needed, and the first K are the row's experts, in rank order. A row with more
// than 32 candidates (all logits equal, as for a row of zeros) or a logit that is not finite (an x beyond f16's range)
// has every logit recomputed exactly instead.
__device__ __forceinline__ void router_topk_row(uint32_t t, const float *rl, const RouterApprox &ap, const float *__restrict__ bias,
                                                uint32_t NE, uint32_t K, int32_t *__restrict__ ids, float *__restrict__ w,
                                                float *__restrict__ gs, uint32_t *hist, int32_t *s_ids, uint8_t *ex_buf) {
  auto exact4 = [&](const float *xr, uint32_t e, uint32_t n, uint32_t ln) {
    return ex_buf ? exact_logits4_staged(xr, ap.W, bias, ap.E, e, n, ln, ex_buf) : exact_logits4(xr, ap.W, bias, ap.E, e, ln);
  };
  const uint32_t lane = threadIdx.x % 32, per = NE / 32;
  uint32_t key[kMaxPerLane];
  float mx = -INFINITY, eps2 = 0.0f;  // eps2: twice the row's error bound; 0 with exact logits
  bool finite = true;
  if (ap.logits) {
    // The row itself is wanted only if some logits have to be recomputed, but then at once: ask for it now.
    const char *row = (const char *)(ap.x + (uint64_t)t * ap.E);
    for (uint32_t b = lane * 128; b < ap.E * 4; b += 32 * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + b));
  }
  // All of the lane's logits are asked for before any is used.
  float f[kMaxPerLane];
  float *const at = ap.logits + (uint64_t)t * NE + lane;
#pragma unroll
  for (int j = 0; j < kMaxPerLane; j++)
    if ((uint32_t)j < per) f[j] = ap.logits ? at[32 * j] : rl[(uint64_t)t * (NE + 1) + lane + 32 * j];
  if (ap.logits && ap.parts > 1) {
    for (uint32_t p = 1; p < ap.parts; p++) {
      float more[kMaxPerLane];
#pragma unroll
      for (int j = 0; j < kMaxPerLane; j++)
        if ((uint32_t)j < per) more[j] = at[p * ap.part_stride + 32 * j];
#pragma unroll
      for (int j = 0; j < kMaxPerLane; j++)
        if ((uint32_t)j < per) f[j] += more[j];
    }
#pragma unroll
    for (int j = 0; j < kMaxPerLane; j++)
      if ((uint32_t)j < per) at[32 * j] = f[j];
  }
#pragma unroll
  for (int j = 0; j < kMaxPerLane; j++) {
    key[j] = 0;
    if ((uint32_t)j < per) {
      if (ap.logits) {
        if (bias) f[j] = __fadd_rn(f[j], bias[lane + 32 * j]);
        finite = finite && isfinite(f[j]);
      }
      key[j] = order_key(f[j]);
      mx = fmaxf(mx, f[j]);
    }
  }
  if (ap.logits) {
    float n2 = 0.0f;
    for (uint32_t p = lane; p < ap.nparts; p += 32) n2 += ap.norm2_parts[(uint64_t)t * ap.nparts + p];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, off);
    eps2 = 2.0f * (ap.eps_rel * sqrtf(n2) + ap.eps_abs);
    finite = __all_sync(0xffffffffu, finite) && isfinite(eps2);
  }
  // Lane k keeps the k-th winner of the rounds below.
  float my_v = 0.0f, sum = 0.0f;
  uint32_t my_id = 0, ncand = 0;
  for (bool exact_all = ap.logits && !finite;;) {
    if (exact_all) {
      // Every logit exactly, four experts a pass: for rows the approximate ones cannot serve.
      mx = -INFINITY;
      for (uint32_t e0 = 0; e0 < NE; e0 += 4) {
        const float v = exact4(ap.x + (uint64_t)t * ap.E, e0 + lane / 8, 4, lane);
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const float vq = __shfl_sync(0xffffffffu, v, 8 * q);
          const uint32_t e = e0 + q;
          if (e % 32 == lane) {
#pragma unroll
            for (int j = 0; j < kMaxPerLane; j++)
              if ((uint32_t)j == e / 32) key[j] = order_key(vq);
          }
          mx = fmaxf(mx, vq);
        }
      }
      eps2 = 0.0f;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    sum = 0.0f;
    if (w) {
#pragma unroll
      for (int j = 0; j < kMaxPerLane; j++)
        if ((uint32_t)j < per) sum += expf(key_value(key[j]) - mx);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    }
    // Rounds of arg-max over (key, lower expert first), which use the keys up. K rounds with exact logits; with
    // approximate ones, on until the next is more than 2 eps below the K-th (at most 32 in all).
    float vK = 0.0f;
    bool overflow = false;
    ncand = 0;
    // A lane keeps the best of its own keys (the lower expert among equals); a round is then two warp reductions,
    // the largest key and among its holders the lowest expert, and only the winner's lane has a new best to find.
    uint32_t lkey = 0, lj = 0;
    auto rescan = [&]() {
      lkey = 0, lj = 0;
#pragma unroll
      for (int j = 0; j < kMaxPerLane; j++)
        if ((uint32_t)j < per && key[j] > lkey) lkey = key[j], lj = j;
    };
    rescan();
    for (uint32_t k = 0; k < 32; k++) {
      const uint32_t bkey = __reduce_max_sync(0xffffffffu, lkey);
      if (bkey == 0) break;  // nothing left (fewer than 32 experts in all)
      const uint32_t e = __reduce_min_sync(0xffffffffu, lkey == bkey ? lane + 32 * lj : 0xFFFFFFFFu);
      const float v = key_value(bkey);
      if (k == K - 1) vK = v;
      if (k >= K && !(eps2 > 0.0f && v >= vK - eps2)) break;
      if (e % 32 == lane) {
#pragma unroll
        for (int j = 0; j < kMaxPerLane; j++)
          if ((uint32_t)j == e / 32) key[j] = 0;
        rescan();
      }
      if (lane == k) my_id = e, my_v = v;
      ncand = k + 1;
      if (k == 31 && eps2 > 0.0f && NE > 32) overflow = true;  // there may be more within reach than a warp holds
    }
    if (!overflow) break;
    exact_all = true;
  }
  if (eps2 > 0.0f) {
    // Neighbours too close to order: both get their exact logit, four candidates a pass.
    const float up = __shfl_up_sync(0xffffffffu, my_v, 1), down = __shfl_down_sync(0xffffffffu, my_v, 1);
    const bool need = lane < ncand && ((lane > 0 && up - my_v <= eps2) || (lane + 1 < ncand && my_v - down <= eps2));
    uint32_t todo = __ballot_sync(0xffffffffu, need);
    while (todo) {
      const uint32_t n = min(4u, (uint32_t)__popc(todo));
      uint32_t c[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        c[q] = todo ? (uint32_t)__ffs(todo) - 1 : 0xFFFFFFFFu;
        if (todo) todo &= todo - 1;
      }
      const uint32_t g8 = lane / 8, mine = g8 == 0 ? c[0] : g8 == 1 ? c[1] : g8 == 2 ? c[2] : c[3];
      const uint32_t e = __shfl_sync(0xffffffffu, my_id, mine == 0xFFFFFFFFu ? 0 : mine);
      const float v = exact4(ap.x + (uint64_t)t * ap.E, e, n, lane);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const float vq = __shfl_sync(0xffffffffu, v, 8 * q);
        if (lane == c[q]) my_v = vq + 0.0f;
      }
    }
  }
  if (!w) {  // the experts alone: with exact logits lane k holds the k-th already
    if (lane < min(ncand, K)) s_ids[lane] = (int32_t)my_id;
    return;
  }
  // Rank among the candidates by (logit, lower expert first); with exact logits this is the order they came in.
  uint32_t rank = 0;
  {
    const unsigned long long me = ((unsigned long long)order_key(my_v) << 32) | (uint32_t)~my_id;
    for (uint32_t j = 0; j < ncand; j++) {
      const unsigned long long o = __shfl_sync(0xffffffffu, me, j);
      rank += o > me;
    }
  }
  const bool winner = lane < ncand && rank < K;
  const float pk = winner ? expf(my_v - mx) / sum : 0.0f;
  // The K winners' p added in rank order.
  float tot = 0.0f;
  for (uint32_t k = 0; k < K; k++) {
    const uint32_t src = __ffs(__ballot_sync(0xffffffffu, winner && rank == k)) - 1;
    tot += __shfl_sync(0xffffffffu, pk, src & 31);
  }
  if (winner) {
    ids[(uint64_t)t * K + rank] = (int32_t)my_id;
    w[(uint64_t)t * K + rank] = pk / fmaxf(tot, 6.1035e-5f);
    if (hist) atomicAdd(&hist[my_id], 1u);
    if (s_ids) s_ids[rank] = (int32_t)my_id;
  }
  if (lane == 0) {
    float g;
    if (ap.logits) {
      g = 0.0f;
      for (uint32_t p = 0; p < ap.nparts; p++) g += ap.gate_parts[(uint64_t)t * ap.nparts + p];
    } else {
      g = rl[(uint64_t)t * (NE + 1) + NE];
    }
    gs[t] = 1.0f / (1.0f + expf(-g));
  }
}

}  // namespace moe

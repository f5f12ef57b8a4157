// The activation quantisers' arithmetic: 256 values by a warp, eight consecutive ones a lane, to q8_0 or q8_K
// (the reference's quantize_a8, kernels/include/a8.h:9-16).
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace moe {

// A lane's share of a quantised block of 256 values: its eight codes (8 bytes), the scale of the block they belong to,
// and (q8_K, even lanes) the sum of the 16 codes that start at the lane's first.
struct QuantLane {
  uint2 codes;
  float d;
  int sum16;
};
__device__ __forceinline__ uint32_t pack_codes(int c0, int c1, int c2, int c3) {
  return (uint32_t)(c0 & 0xFF) | (uint32_t)(c1 & 0xFF) << 8 | (uint32_t)(c2 & 0xFF) << 16 | (uint32_t)c3 << 24;
}

// q8_0: per 32 values d = max|x| / 127, q = round(x * (1 / d)), 0 when d is 0; d kept as the f16 the CPU stores
// (docs/spec/QUANT_FORMATS.md:463-465, :525-526).
// q8_K: per 256 values iscale = -127 / max with max the value of largest magnitude (the first of equals),
// q = min(127, nearest-even(iscale * x)), d = 1 / iscale, and the sums of each 16 codes (QUANT_FORMATS.md:528-535).
template <bool Q8K>
__device__ __forceinline__ QuantLane quantize_lane(const float4 &a, const float4 &b, uint32_t lane) {
  const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  QuantLane o{};
  int c[8];
  if constexpr (!Q8K) {
    float amax = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))),
                       fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fmaxf(fabsf(b.z), fabsf(b.w))));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));  // 4 lanes hold a block of 32
    const float dd = amax / 127.0f, id = dd != 0.0f ? 1.0f / dd : 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) c[i] = (signed char)roundf(v[i] * id);
    o.d = __half2float(__float2half_rn(dd));
  } else {
    float amax = 0.0f, mx = 0.0f;
    uint32_t at = 8 * lane;
#pragma unroll
    for (int i = 0; i < 8; i++)
      if (fabsf(v[i]) > amax) amax = fabsf(v[i]), mx = v[i], at = 8 * lane + i;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const float oa = __shfl_xor_sync(0xffffffffu, amax, off), om = __shfl_xor_sync(0xffffffffu, mx, off);
      const uint32_t oat = __shfl_xor_sync(0xffffffffu, at, off);
      if (oa > amax || (oa == amax && oat < at)) amax = oa, mx = om, at = oat;
    }
    if (amax == 0.0f) return o;  // the same for the whole warp: codes, scale and sums 0
    const float iscale = -127.0f / mx;
    int sum = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) c[i] = min(127, __float2int_rn(__fmul_rn(iscale, v[i]))), sum += c[i];
    o.sum16 = sum + __shfl_xor_sync(0xffffffffu, sum, 1);
    o.d = 1.0f / iscale;
  }
  o.codes = make_uint2(pack_codes(c[0], c[1], c[2], c[3]), pack_codes(c[4], c[5], c[6], c[7]));
  return o;
}

// Eight codes dequantised, f16: what the tensor-core kernels take for a row.
__device__ __forceinline__ uint4 dequant_lane(const QuantLane &o) {
  uint4 r;
  uint32_t *p = &r.x;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint32_t w = (i < 2 ? o.codes.x : o.codes.y) >> (16 * (i & 1));
    const __half2 h = __floats2half2_rn(o.d * (float)(signed char)(w & 0xFF), o.d * (float)(signed char)((w >> 8) & 0xFF));
    p[i] = *(const uint32_t *)&h;
  }
  return r;
}

// Where a quantised buffer's rows go: codes, scales, q8_K's sums, and the f16 form (null: not wanted). q null: no job.
struct QuantJob {
  int8_t *q;
  float *d;
  int16_t *bs;
  __half *deq;
  uint32_t q8k;
};
// A lane's share of block blk into job's codes, scales and sums.
template <bool Q8K>
__device__ __forceinline__ void store_codes(const QuantLane &o, uint64_t blk, uint32_t lane, const QuantJob &job) {
  ((uint2 *)(job.q + blk * 256))[lane] = o.codes;
  if constexpr (Q8K) {
    if (lane == 0) job.d[blk] = o.d;
    if (lane % 2 == 0) job.bs[blk * 16 + lane / 2] = (int16_t)o.sum16;
  } else {
    if (lane % 4 == 0) job.d[blk * 8 + lane / 4] = o.d;
  }
}
// Block blk of 256 values, held eight a lane, into job's buffers.
template <bool Q8K>
__device__ __forceinline__ void quantize_store(const float4 &a, const float4 &b, uint64_t blk, uint32_t lane, const QuantJob &job) {
  const QuantLane o = quantize_lane<Q8K>(a, b, lane);
  store_codes<Q8K>(o, blk, lane, job);
  if (job.deq) ((uint4 *)(job.deq + blk * 256))[lane] = dequant_lane(o);
}

}  // namespace moe

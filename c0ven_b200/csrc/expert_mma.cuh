// The experts' products for a few rows per expert (up to 32), exact as the integer-dot kernels are: the weights' codes as
// int8 against the rows' int8 codes on the warp-level tensor instruction (mma.sync, int8 in, int32 out), 16 weight rows
// by 8 activation rows an instruction, one sub-block of the weights (32 values, or 16 where the type scales 16) at
// a time; the integer sums then meet the sub-block's scale in int32 and the block's in f32, as the CPU path's dots do
// (core/cpu/experts.cpp:152-284).
//
// Why this unit and not tcgen05: its sums would leave tensor memory once per sub-block to be scaled, so the tile kernel
// decodes to f16 with the scales folded in, some 5.5 instructions a weight, and with a dozen rows an expert that decode is
// the whole of its time. Here a weight stays the code it is: for Q4_K an AND (and a shift) a word of eight, and 3.6
// instructions a weight with 15 rows, multiply-adds, scales and all (counted: 119.7 million warp instructions for gate and
// up of 777 rows). The rows' codes are read from shared memory at one word per lane a sub-block, where dp4a needs a 16-byte
// piece per lane and row. What bounds it is the wait for a warp's next block of weights, at two CTAs an SM (Q8_0, 100 rows:
// 4.5 TB/s, issue slots a third busy), and with more rows the instructions beside it.
//
// A warp takes 16 weight rows at a time over the whole row length, from registers, a block of 256 values ahead; which of a
// sub-block's values sit in which lane is free as long as both operands agree, and is chosen so that a lane's share of a
// sub-block is contiguous in memory.
#pragma once

#include "expert_rows.cuh"

namespace moe {

constexpr uint32_t kMmaRows = 32;               // activation rows an entry holds at most
constexpr uint32_t kMmaCtaRows = 8 * 16;        // weight rows a CTA takes at a time: 16 a warp
constexpr uint32_t kMmaMaxSmem = 100 * 1024;    // two CTAs an SM

// The rows in shared memory: codes with a stride that spreads eight rows' words over the banks; the scales, sub-block or
// block by block with the rows side by side; the sums of each 32 or 16 codes. After them a codebook type's codebook.
__host__ __device__ constexpr uint32_t mma_pad(uint32_t qt) { return qt == QT_Q6_K || qt == QT_IQ4_NL || qt == QT_IQ4_XS || qt == QT_IQ2_S ? 16 : 32; }
__host__ __device__ constexpr uint32_t mma_sum_len(uint32_t qt) { return qt == QT_Q4_K ? 32 : qt == QT_Q6_K ? 16 : 0; }
__host__ __device__ constexpr uint32_t mma_smem(uint32_t qt, uint32_t rows, uint32_t K) {
  const uint32_t sums = mma_sum_len(qt) ? K / mma_sum_len(qt) * 2 + 16 : 0;
  return rows * (K + mma_pad(qt)) + rows * (act_is_q8k(qt) ? K / 256 : K / 32) * 4 + rows * sums + 4 * grid_words(qt);
}
// Whether the kernel takes entries of up to `rows` rows (8 or kMmaRows) of K values: a CTA holds them all.
__host__ __device__ constexpr bool mma_takes(uint32_t qt, uint32_t K, uint32_t rows) {
  return K % 256 == 0 && mma_smem(qt, rows, K) <= kMmaMaxSmem;
}

// Whether a warp loads a block ahead of the one it multiplies. The codebook types hold so much of a block that a second one
// spills at two CTAs an SM; without it three fit, and the other warps cover the wait (13 rows of IQ2_S 172 -> 160 us, 200
// of IQ3_S 504 -> 491).
__host__ __device__ constexpr bool mma_ahead(uint32_t qt) { return grid_words(qt) == 0; }

struct ExpertMmaArgs {
  const uint8_t *w0, *w1;   // slot 0's slice of (gate, up) or (down, unused), runs layout
  uint64_t slice_bytes;
  uint32_t K, R;            // values per weight row; weight rows (a multiple of 128)
  ActView act;
  const uint32_t *act_row;  // expert-order row -> activation row; null: the same row
  const MoeGroup *entries;  // (slot, start, n), n <= kMmaRows: the list's entries *first .. *end
  const uint32_t *first, *end;
  const MoeGroup *entries2; // after them, entries 0 .. *end2 of a second list; either list may be left out (end null)
  const uint32_t *end2;
  uint32_t slabs;           // slabs of kMmaCtaRows weight rows a CTA takes one after another
  void *out;                // out[expert-order row][r]: f32, or f16 when out_f16 is set
  uint32_t out_stride, out_f16;
  float limit;
  const uint32_t *grid;     // the codebooks (formats.h: grid_offset)
};

__device__ __forceinline__ void mma_k32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
               : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
               : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
               : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
__device__ __forceinline__ uint2 ldg_stream8(const void *p) {
  uint2 v;
  asm volatile("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ int dp2a_lo(uint32_t s16x2, uint32_t b8x4, int c) {
  int d;
  asm("dp2a.lo.s32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(s16x2), "r"(b8x4), "r"(c));
  return d;
}
__device__ __forceinline__ int dp2a_hi(uint32_t s16x2, uint32_t b8x4, int c) {
  int d;
  asm("dp2a.hi.s32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(s16x2), "r"(b8x4), "r"(c));
  return d;
}
__device__ __forceinline__ int sbyte(uint32_t w, int i) { return (int)(w << (24 - 8 * i)) >> 24; }

// What a block's product reads of the rows: codes of row n at codes + n * stride; scales, NT * 8 rows side by side; sums of
// row n at sums + n * sum_stride (int16).
struct MmaActs {
  const uint8_t *codes;
  const float *scales;
  const int16_t *sums;
  uint32_t stride, sum_stride;
  const uint32_t *grid;  // a codebook type's codebook
};

// A type's share of a lane: Row is what it holds of one weight row's block of 256 values (lane j = lane % 4 of the four that
// share the row); block() adds the products of two weight rows (g and g + 8 of the warp's 16, g = lane / 4) with columns
// 2 j, 2 j + 1 of each of the NT tiles of 8 activation rows to f.
template <int QT>
struct Frag;

// Q4_K: y = d * sc * q - dmin * m. A pair of sub-blocks is 32 bytes, their low and high nibbles; a lane's share 8 of them:
// values 8 j .. 8 j + 7 of either sub-block.
template <>
struct Frag<QT_Q4_K> {
  struct Row {
    uint2 q[4];
    uint4 hd;
  };
  __device__ static __forceinline__ Row fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t b, uint32_t j) {
    Row x;
    const uint64_t blk = (uint64_t)r * (K / 256) + b;
#pragma unroll
    for (int p = 0; p < 4; p++) x.q[p] = ldg_stream8(s + 128 * blk + 32 * p + 8 * j);
    x.hd = __ldg((const uint4 *)(s + 128 * nblk + 16 * blk));
    return x;
  }
  // The eight 6-bit scales and minimums as bytes (QUANT_FORMATS.md:386-392).
  __device__ static __forceinline__ void scales(const uint4 &hd, uint32_t (&sc)[2], uint32_t (&mn)[2]) {
    sc[0] = hd.y & 0x3F3F3F3Fu, mn[0] = hd.z & 0x3F3F3F3Fu;
    sc[1] = (hd.w & 0x0F0F0F0Fu) | ((hd.y >> 2) & 0x30303030u), mn[1] = ((hd.w >> 4) & 0x0F0F0F0Fu) | ((hd.z >> 2) & 0x30303030u);
  }
  template <int NT>
  __device__ static __forceinline__ void block(const Row &x, const Row &y, uint32_t b, uint32_t g, uint32_t j, const MmaActs &acts, float (&f)[NT][4]) {
    uint32_t scx[2], mnx[2], scy[2], mny[2];
    scales(x.hd, scx, mnx), scales(y.hd, scy, mny);
    int sum[NT][4];
#pragma unroll
    for (int t = 0; t < NT; t++) sum[t][0] = sum[t][1] = sum[t][2] = sum[t][3] = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint2 qx = x.q[i / 2], qy = y.q[i / 2];
      const int sh = 4 * (i & 1), sx = sbyte(scx[i / 4], i & 3), sy = sbyte(scy[i / 4], i & 3);
      const uint32_t a0 = (qx.x >> sh) & 0x0F0F0F0Fu, a2 = (qx.y >> sh) & 0x0F0F0F0Fu, a1 = (qy.x >> sh) & 0x0F0F0F0Fu, a3 = (qy.y >> sh) & 0x0F0F0F0Fu;
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const uint2 v = *(const uint2 *)(acts.codes + (8 * t + g) * acts.stride + 256 * b + 32 * i + 8 * j);
        int c[4];
        mma_k32(c, a0, a1, a2, a3, v.x, v.y);
        sum[t][0] += sx * c[0], sum[t][1] += sx * c[1], sum[t][2] += sy * c[2], sum[t][3] += sy * c[3];
      }
    }
    const float2 dx = __half22float2(*(const __half2 *)&x.hd.x), dy = __half22float2(*(const __half2 *)&y.hd.x);  // d, dmin
#pragma unroll
    for (int t = 0; t < NT; t++) {
      const float2 da = *(const float2 *)(acts.scales + b * 8 * NT + 8 * t + 2 * j);
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const uint4 s = *(const uint4 *)(acts.sums + (8 * t + 2 * j + k) * acts.sum_stride + 8 * b);
        const int mx = dp2a_hi(s.w, mnx[1], dp2a_lo(s.z, mnx[1], dp2a_hi(s.y, mnx[0], dp2a_lo(s.x, mnx[0], 0))));
        const int my = dp2a_hi(s.w, mny[1], dp2a_lo(s.z, mny[1], dp2a_hi(s.y, mny[0], dp2a_lo(s.x, mny[0], 0))));
        const float d = k ? da.y : da.x;
        f[t][k] += d * (dx.x * (float)sum[t][k] - dx.y * (float)mx);
        f[t][2 + k] += d * (dy.x * (float)sum[t][2 + k] - dy.y * (float)my);
      }
    }
  }
};

// Q8_0: y = d * q, eight blocks of 32 with a scale each, as the rows' codes have. A lane's share of a block: 8 bytes.
template <>
struct Frag<QT_Q8_0> {
  struct Row {
    uint2 q[8];
    uint4 d;
  };
  __device__ static __forceinline__ Row fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t b, uint32_t j) {
    Row x;
    const uint8_t *q = s + (uint64_t)r * K + 256 * b + 8 * j;
#pragma unroll
    for (int i = 0; i < 8; i++) x.q[i] = ldg_stream8(q + 32 * i);
    x.d = __ldg((const uint4 *)((const __half *)(s + 32 * nblk) + (uint64_t)r * (K / 32) + 8 * b));
    return x;
  }
  __device__ static __forceinline__ float scale(const uint4 &d, int i) {
    const uint32_t w = i < 2 ? d.x : i < 4 ? d.y : i < 6 ? d.z : d.w;
    const __half2 h = *(const __half2 *)&w;
    return i & 1 ? __high2float(h) : __low2float(h);
  }
  template <int NT>
  __device__ static __forceinline__ void block(const Row &x, const Row &y, uint32_t b, uint32_t g, uint32_t j, const MmaActs &acts, float (&f)[NT][4]) {
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const float dx = scale(x.d, i), dy = scale(y.d, i);
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const uint2 v = *(const uint2 *)(acts.codes + (8 * t + g) * acts.stride + 256 * b + 32 * i + 8 * j);
        const float2 da = *(const float2 *)(acts.scales + (8 * b + i) * 8 * NT + 8 * t + 2 * j);
        int c[4];
        mma_k32(c, x.q[i].x, y.q[i].x, x.q[i].y, y.q[i].y, v.x, v.y);
        f[t][0] = fmaf(dx * da.x, (float)c[0], f[t][0]), f[t][1] = fmaf(dx * da.y, (float)c[1], f[t][1]);
        f[t][2] = fmaf(dy * da.x, (float)c[2], f[t][2]), f[t][3] = fmaf(dy * da.y, (float)c[3], f[t][3]);
      }
    }
  }
};

// Q6_K: y = d * scales[v / 16] * (q - 32), 16 values a scale. Of each 16 a lane's share is four: a word of ql (its low or
// its high nibbles) and two bits a byte of qh. The 32 comes out through the sums of the rows' codes.
template <>
struct Frag<QT_Q6_K> {
  struct Row {
    uint32_t l[8], h[4];
    uint4 sc;
    float d;
  };
  __device__ static __forceinline__ Row fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t b, uint32_t j) {
    Row x;
    const uint64_t blk = (uint64_t)r * (K / 256) + b;
#pragma unroll
    for (int i = 0; i < 8; i++) x.l[i] = __ldg((const uint32_t *)(s + 128 * blk + 16 * i) + j);
#pragma unroll
    for (int i = 0; i < 4; i++) x.h[i] = __ldg((const uint32_t *)(s + 128 * nblk + 64 * blk + 16 * i) + j);
    x.sc = __ldg((const uint4 *)(s + 192 * nblk + 16 * blk));
    x.d = __half2float(__ldg((const __half *)(s + 208 * nblk) + blk));
    return x;
  }
  // The codes of group i of 16 values, 0 .. 63: half i / 8, quarter (i / 2) % 4 of it, its 16 bytes i % 2.
  __device__ static __forceinline__ uint32_t codes(const Row &x, int i) {
    const int hh = i / 8, qr = (i / 2) % 4, hb = i % 2;
    return ((x.l[4 * hh + 2 * (qr & 1) + hb] >> (4 * (qr >> 1))) & 0x0F0F0F0Fu) | (((x.h[2 * hh + hb] >> (2 * qr)) & 0x03030303u) << 4);
  }
  template <int NT>
  __device__ static __forceinline__ void block(const Row &x, const Row &y, uint32_t b, uint32_t g, uint32_t j, const MmaActs &acts, float (&f)[NT][4]) {
    const uint32_t scx[4] = {x.sc.x, x.sc.y, x.sc.z, x.sc.w}, scy[4] = {y.sc.x, y.sc.y, y.sc.z, y.sc.w};
    int sum[NT][4];
#pragma unroll
    for (int t = 0; t < NT; t++) sum[t][0] = sum[t][1] = sum[t][2] = sum[t][3] = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const uint32_t a0 = codes(x, i), a1 = codes(y, i);
      const int sx = sbyte(scx[i / 4], i & 3), sy = sbyte(scy[i / 4], i & 3);
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const uint32_t v = *(const uint32_t *)(acts.codes + (8 * t + g) * acts.stride + 256 * b + 16 * i + 4 * j);
        int c[4];
        mma_k16(c, a0, a1, v);
        sum[t][0] += sx * c[0], sum[t][1] += sx * c[1], sum[t][2] += sy * c[2], sum[t][3] += sy * c[3];
      }
    }
#pragma unroll
    for (int t = 0; t < NT; t++) {
      const float2 da = *(const float2 *)(acts.scales + b * 8 * NT + 8 * t + 2 * j);
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const uint4 *s = (const uint4 *)(acts.sums + (8 * t + 2 * j + k) * acts.sum_stride + 16 * b);
        const uint4 s0 = s[0], s1 = s[1];
        const uint32_t sm[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
        int mx = 0, my = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          mx = dp2a_hi(sm[2 * q + 1], scx[q], dp2a_lo(sm[2 * q], scx[q], mx));
          my = dp2a_hi(sm[2 * q + 1], scy[q], dp2a_lo(sm[2 * q], scy[q], my));
        }
        const float d = k ? da.y : da.x;
        f[t][k] = fmaf(x.d * d, (float)(sum[t][k] - 32 * mx), f[t][k]);
        f[t][2 + k] = fmaf(y.d * d, (float)(sum[t][2 + k] - 32 * my), f[t][2 + k]);
      }
    }
  }
};

// IQ4_XS and IQ4_NL: 16 bytes hold a sub-block's values 0 .. 15 in their low nibbles and 16 .. 31 in their high ones; a
// lane's share is four bytes, values 4 j .. and 16 + 4 j .., through the table.
struct FragIq4 {
  __device__ static __forceinline__ void mma(int (&c)[4], const uint32_t *x, const uint32_t *y, const uint8_t *v) {
    mma_k32(c, x[0], y[0], x[1], y[1], *(const uint32_t *)v, *(const uint32_t *)(v + 16));
  }
};
// y = d * (ls - 32) * table[q], a 6-bit ls a sub-block.
template <>
struct Frag<QT_IQ4_XS> {
  struct Row {
    uint32_t q[8], sl, sh;
    float d;
  };
  __device__ static __forceinline__ Row fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t b, uint32_t j) {
    Row x;
    const uint64_t blk = (uint64_t)r * (K / 256) + b;
#pragma unroll
    for (int i = 0; i < 8; i++) x.q[i] = __ldg((const uint32_t *)(s + 128 * blk + 16 * i) + j);
    x.sl = __ldg((const uint32_t *)(s + 128 * nblk) + blk), x.sh = __ldg((const uint16_t *)(s + 132 * nblk) + blk);
    x.d = __half2float(__ldg((const __half *)(s + 134 * nblk) + blk));
    return x;
  }
  template <int NT>
  __device__ static __forceinline__ void block(const Row &x, const Row &y, uint32_t b, uint32_t g, uint32_t j, const MmaActs &acts, float (&f)[NT][4]) {
    int sum[NT][4];
#pragma unroll
    for (int t = 0; t < NT; t++) sum[t][0] = sum[t][1] = sum[t][2] = sum[t][3] = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      uint32_t a[2], c2[2];
      iq4_lookup8(x.q[i], a[0], a[1]), iq4_lookup8(y.q[i], c2[0], c2[1]);
      const int sx = (int)(((x.sl >> (4 * i)) & 0xF) | (((x.sh >> (2 * i)) & 3) << 4)) - 32, sy = (int)(((y.sl >> (4 * i)) & 0xF) | (((y.sh >> (2 * i)) & 3) << 4)) - 32;
#pragma unroll
      for (int t = 0; t < NT; t++) {
        int c[4];
        FragIq4::mma(c, a, c2, acts.codes + (8 * t + g) * acts.stride + 256 * b + 32 * i + 4 * j);
        sum[t][0] += sx * c[0], sum[t][1] += sx * c[1], sum[t][2] += sy * c[2], sum[t][3] += sy * c[3];
      }
    }
#pragma unroll
    for (int t = 0; t < NT; t++) {
      const float2 da = *(const float2 *)(acts.scales + b * 8 * NT + 8 * t + 2 * j);
      f[t][0] = fmaf(x.d * da.x, (float)sum[t][0], f[t][0]), f[t][1] = fmaf(x.d * da.y, (float)sum[t][1], f[t][1]);
      f[t][2] = fmaf(y.d * da.x, (float)sum[t][2], f[t][2]), f[t][3] = fmaf(y.d * da.y, (float)sum[t][3], f[t][3]);
    }
  }
};
// y = d * table[q], a scale a block of 32.
template <>
struct Frag<QT_IQ4_NL> {
  struct Row {
    uint32_t q[8];
    uint4 d;
  };
  __device__ static __forceinline__ Row fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t b, uint32_t j) {
    Row x;
#pragma unroll
    for (int i = 0; i < 8; i++) x.q[i] = __ldg((const uint32_t *)(s + (uint64_t)r * (K / 2) + 128 * b + 16 * i) + j);
    x.d = __ldg((const uint4 *)((const __half *)(s + 16 * nblk) + (uint64_t)r * (K / 32) + 8 * b));
    return x;
  }
  template <int NT>
  __device__ static __forceinline__ void block(const Row &x, const Row &y, uint32_t b, uint32_t g, uint32_t j, const MmaActs &acts, float (&f)[NT][4]) {
#pragma unroll
    for (int i = 0; i < 8; i++) {
      uint32_t a[2], c2[2];
      iq4_lookup8(x.q[i], a[0], a[1]), iq4_lookup8(y.q[i], c2[0], c2[1]);
      const float dx = Frag<QT_Q8_0>::scale(x.d, i), dy = Frag<QT_Q8_0>::scale(y.d, i);
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const float2 da = *(const float2 *)(acts.scales + (8 * b + i) * 8 * NT + 8 * t + 2 * j);
        int c[4];
        FragIq4::mma(c, a, c2, acts.codes + (8 * t + g) * acts.stride + 256 * b + 32 * i + 4 * j);
        f[t][0] = fmaf(dx * da.x, (float)c[0], f[t][0]), f[t][1] = fmaf(dx * da.y, (float)c[1], f[t][1]);
        f[t][2] = fmaf(dy * da.x, (float)c[2], f[t][2]), f[t][3] = fmaf(dy * da.y, (float)c[3], f[t][3]);
      }
    }
  }
};

// The two bytes that are lane j's share of sub-block i (8 bytes), where lane j of the four loaded the 16 bytes of sub-blocks
// 2 j and 2 j + 1: one wide load a row in place of eight narrow ones, and two shuffles a sub-block.
__device__ __forceinline__ uint32_t quad_share(const uint4 &q, int i, uint32_t j) {
  const uint32_t w0 = __shfl_sync(0xffffffffu, i & 1 ? q.z : q.x, i / 2, 4), w1 = __shfl_sync(0xffffffffu, i & 1 ? q.w : q.y, i / 2, 4);
  return (j & 2 ? w1 : w0) >> (16 * (j & 1));
}
__device__ __forceinline__ uint32_t word_of(const uint4 (&v)[2], int i) {
  const uint4 &u = v[i / 4];
  return (i & 3) == 0 ? u.x : (i & 3) == 1 ? u.y : (i & 3) == 2 ? u.z : u.w;
}
__device__ __forceinline__ uint32_t byte_of(const uint2 &v, int i) { return ((i < 4 ? v.x : v.y) >> (8 * (i & 3))) & 0xFF; }

// Sub-blocks of 32 with an integer scale each and one f32 scale a block: codebook types whose lane's share of a sub-block
// is two words of four values, 8 j .. 8 j + 7. WORDS(row, i, j, grid, a) leaves them in a, SCALE(row, i) is the scale.
template <class Type, int NT>
__device__ __forceinline__ void block_of_words(const typename Type::Row &x, const typename Type::Row &y, uint32_t b, uint32_t g, uint32_t j,
                                               const MmaActs &acts, float (&f)[NT][4]) {
  int sum[NT][4];
#pragma unroll
  for (int t = 0; t < NT; t++) sum[t][0] = sum[t][1] = sum[t][2] = sum[t][3] = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    uint32_t ax[2], ay[2];
    Type::words(x, i, j, acts.grid, ax), Type::words(y, i, j, acts.grid, ay);
    const int sx = Type::scale(x, i), sy = Type::scale(y, i);
#pragma unroll
    for (int t = 0; t < NT; t++) {
      const uint2 v = *(const uint2 *)(acts.codes + (8 * t + g) * acts.stride + 256 * b + 32 * i + 8 * j);
      int c[4];
      mma_k32(c, ax[0], ay[0], ax[1], ay[1], v.x, v.y);
      sum[t][0] += sx * c[0], sum[t][1] += sx * c[1], sum[t][2] += sy * c[2], sum[t][3] += sy * c[3];
    }
  }
#pragma unroll
  for (int t = 0; t < NT; t++) {
    const float2 da = *(const float2 *)(acts.scales + b * 8 * NT + 8 * t + 2 * j);
    f[t][0] = fmaf(x.d * da.x, (float)sum[t][0], f[t][0]), f[t][1] = fmaf(x.d * da.y, (float)sum[t][1], f[t][1]);
    f[t][2] = fmaf(y.d * da.x, (float)sum[t][2], f[t][2]), f[t][3] = fmaf(y.d * da.y, (float)sum[t][3], f[t][3]);
  }
}

// IQ3_S: y = d * (1 + 2 s) * grid[index][i] * sign, a 9-bit index and a nibble of signs for each four values.
template <>
struct Frag<QT_IQ3_S> {
  struct Row {
    uint4 qs, sg[2];
    uint2 qh;
    uint32_t sc;
    float d;
  };
  __device__ static __forceinline__ Row fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t b, uint32_t j) {
    Row x;
    const uint64_t blk = (uint64_t)r * (K / 256) + b;
    x.qs = __ldg((const uint4 *)(s + 64 * blk) + j);
    x.sg[0] = __ldg((const uint4 *)(s + 64 * nblk + 32 * blk)), x.sg[1] = __ldg((const uint4 *)(s + 64 * nblk + 32 * blk) + 1);
    x.qh = __ldg((const uint2 *)(s + 96 * nblk) + blk);
    x.sc = __ldg((const uint32_t *)(s + 104 * nblk) + blk);
    x.d = __half2float(__ldg((const __half *)(s + 108 * nblk) + blk));
    return x;
  }
  __device__ static __forceinline__ void words(const Row &x, int i, uint32_t j, const uint32_t *grid, uint32_t (&a)[2]) {
    const uint32_t q = quad_share(x.qs, i, j), h = byte_of(x.qh, i) >> (2 * j), sb = word_of(x.sg, i) >> (8 * j);
    a[0] = (uint32_t)signed_word(grid[(q & 0xFF) | ((h & 1u) << 8)], sb & 0xF);
    a[1] = (uint32_t)signed_word(grid[((q >> 8) & 0xFF) | ((h & 2u) << 7)], (sb >> 4) & 0xF);
  }
  __device__ static __forceinline__ int scale(const Row &x, int i) { return 2 * (int)((x.sc >> (4 * i)) & 0xF) + 1; }
  template <int NT>
  __device__ static __forceinline__ void block(const Row &x, const Row &y, uint32_t b, uint32_t g, uint32_t j, const MmaActs &acts, float (&f)[NT][4]) {
    block_of_words<Frag, NT>(x, y, b, g, j, acts, f);
  }
};

// IQ3_XXS: y = d * (0.5 + s) / 2 * grid[index][i] * sign, an 8-bit index for each four values, a 7-bit sign index (the
// eighth sign its parity) for each eight, s in the top four bits of the sub-block's word.
template <>
struct Frag<QT_IQ3_XXS> {
  struct Row {
    uint4 qs, w[2];
    float d;
  };
  __device__ static __forceinline__ Row fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t b, uint32_t j) {
    Row x;
    const uint64_t blk = (uint64_t)r * (K / 256) + b;
    x.qs = __ldg((const uint4 *)(s + 64 * blk) + j);
    x.w[0] = __ldg((const uint4 *)(s + 64 * nblk + 32 * blk)), x.w[1] = __ldg((const uint4 *)(s + 64 * nblk + 32 * blk) + 1);
    x.d = 0.25f * __half2float(__ldg((const __half *)(s + 96 * nblk) + blk));  // (2 s + 1) / 4 = (0.5 + s) / 2
    return x;
  }
  __device__ static __forceinline__ void words(const Row &x, int i, uint32_t j, const uint32_t *grid, uint32_t (&a)[2]) {
    const uint32_t q = quad_share(x.qs, i, j), k7 = (word_of(x.w, i) >> (7 * j)) & 127u, sb = k7 | ((__popc(k7) & 1u) << 7);
    a[0] = (uint32_t)signed_word(grid[q & 0xFF], sb & 0xF), a[1] = (uint32_t)signed_word(grid[(q >> 8) & 0xFF], sb >> 4);
  }
  __device__ static __forceinline__ int scale(const Row &x, int i) { return 2 * (int)(word_of(x.w, i) >> 28) + 1; }
  template <int NT>
  __device__ static __forceinline__ void block(const Row &x, const Row &y, uint32_t b, uint32_t g, uint32_t j, const MmaActs &acts, float (&f)[NT][4]) {
    block_of_words<Frag, NT>(x, y, b, g, j, acts, f);
  }
};

// IQ2_S: y = d * (0.5 + s) / 4 * grid[index][i] * sign, a 10-bit index and a byte of signs for each eight values, an s for
// each 16. A lane's share of 16 values is half an entry: four values, 4 j ..
template <>
struct Frag<QT_IQ2_S> {
  struct Row {
    uint4 qs[2], sg[2];
    uint2 qh, sc;
    float d;
  };
  __device__ static __forceinline__ Row fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t b, uint32_t) {
    Row x;
    const uint64_t blk = (uint64_t)r * (K / 256) + b;
    x.qs[0] = __ldg((const uint4 *)(s + 32 * blk)), x.qs[1] = __ldg((const uint4 *)(s + 32 * blk) + 1);
    x.sg[0] = __ldg((const uint4 *)(s + 32 * nblk + 32 * blk)), x.sg[1] = __ldg((const uint4 *)(s + 32 * nblk + 32 * blk) + 1);
    x.qh = __ldg((const uint2 *)(s + 64 * nblk) + blk), x.sc = __ldg((const uint2 *)(s + 72 * nblk) + blk);
    x.d = 0.125f * __half2float(__ldg((const __half *)(s + 80 * nblk) + blk));  // (2 s + 1) / 8 = (0.5 + s) / 4
    return x;
  }
  __device__ static __forceinline__ uint32_t word(const Row &x, int i, int h, uint32_t j, const uint32_t *grid) {
    const uint32_t e = 2 * h + j / 2;  // the entry within the sub-block
    const uint32_t idx = ((word_of(x.qs, i) >> (8 * e)) & 0xFF) | (((byte_of(x.qh, i) >> (2 * e)) & 3u) << 8);
    return (uint32_t)signed_word(grid[2 * idx + (j & 1)], (word_of(x.sg, i) >> (8 * e + 4 * (j & 1))) & 0xF);
  }
  template <int NT>
  __device__ static __forceinline__ void block(const Row &x, const Row &y, uint32_t b, uint32_t g, uint32_t j, const MmaActs &acts, float (&f)[NT][4]) {
    int sum[NT][4];
#pragma unroll
    for (int t = 0; t < NT; t++) sum[t][0] = sum[t][1] = sum[t][2] = sum[t][3] = 0;
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const uint32_t a0 = word(x, i, h, j, acts.grid), a1 = word(y, i, h, j, acts.grid);
        const int sx = 2 * (int)((byte_of(x.sc, i) >> (4 * h)) & 0xF) + 1, sy = 2 * (int)((byte_of(y.sc, i) >> (4 * h)) & 0xF) + 1;
#pragma unroll
        for (int t = 0; t < NT; t++) {
          int c[4];
          mma_k16(c, a0, a1, *(const uint32_t *)(acts.codes + (8 * t + g) * acts.stride + 256 * b + 32 * i + 16 * h + 4 * j));
          sum[t][0] += sx * c[0], sum[t][1] += sx * c[1], sum[t][2] += sy * c[2], sum[t][3] += sy * c[3];
        }
      }
#pragma unroll
    for (int t = 0; t < NT; t++) {
      const float2 da = *(const float2 *)(acts.scales + b * 8 * NT + 8 * t + 2 * j);
      f[t][0] = fmaf(x.d * da.x, (float)sum[t][0], f[t][0]), f[t][1] = fmaf(x.d * da.y, (float)sum[t][1], f[t][1]);
      f[t][2] = fmaf(y.d * da.x, (float)sum[t][2], f[t][2]), f[t][3] = fmaf(y.d * da.y, (float)sum[t][3], f[t][3]);
    }
  }
};

// Q2_0: y = (q - 1) * d, a scale for each 64 values (the rows': 32); four values a byte.
template <>
struct Frag<QT_Q2_0> {
  struct Row {
    uint4 q;
    uint2 d;
  };
  __device__ static __forceinline__ Row fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t b, uint32_t j) {
    Row x;
    x.q = __ldg((const uint4 *)(s + (uint64_t)r * (K / 4) + 64 * b) + j);
    x.d = __ldg((const uint2 *)((const __half *)(s + 16 * nblk) + (uint64_t)r * (K / 64) + 4 * b));
    return x;
  }
  __device__ static __forceinline__ float scale(const uint2 &d, int i) {
    const uint32_t w = i < 4 ? d.x : d.y;
    const __half2 h = *(const __half2 *)&w;
    return i & 2 ? __high2float(h) : __low2float(h);
  }
  template <int NT>
  __device__ static __forceinline__ void block(const Row &x, const Row &y, uint32_t b, uint32_t g, uint32_t j, const MmaActs &acts, float (&f)[NT][4]) {
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t qx = quad_share(x.q, i, j), qy = quad_share(y.q, i, j);
      const uint32_t a0 = q2_bytes(qx & 0xFF), a2 = q2_bytes((qx >> 8) & 0xFF), a1 = q2_bytes(qy & 0xFF), a3 = q2_bytes((qy >> 8) & 0xFF);
      const float dx = scale(x.d, i), dy = scale(y.d, i);
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const uint2 v = *(const uint2 *)(acts.codes + (8 * t + g) * acts.stride + 256 * b + 32 * i + 8 * j);
        const float2 da = *(const float2 *)(acts.scales + (8 * b + i) * 8 * NT + 8 * t + 2 * j);
        int c[4];
        mma_k32(c, a0, a1, a2, a3, v.x, v.y);
        f[t][0] = fmaf(dx * da.x, (float)c[0], f[t][0]), f[t][1] = fmaf(dx * da.y, (float)c[1], f[t][1]);
        f[t][2] = fmaf(dy * da.x, (float)c[2], f[t][2]), f[t][3] = fmaf(dy * da.y, (float)c[3], f[t][3]);
      }
    }
  }
};

// A CTA's part of an entry whose rows fill NT tiles of 8.
template <int QT, int NMAT, int NT>
__device__ __forceinline__ void mma_entry(const ExpertMmaArgs &a, const MoeGroup &en, uint8_t *smem) {
  constexpr bool q8k = act_is_q8k(QT);
  constexpr uint32_t SL = mma_sum_len(QT);
  const uint32_t K = a.K, n = en.n, start = en.start, KB = K / 256, per_row = q8k ? KB : K / 32;
  const uint64_t nblk = (uint64_t)a.R * (K / block_values(QT));
  const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32, g = lane / 4, j = lane % 4;
  const uint8_t *w[2] = {a.w0 + (uint64_t)en.slot * a.slice_bytes, NMAT == 2 ? a.w1 + (uint64_t)en.slot * a.slice_bytes : nullptr};
  const uint32_t r_first = blockIdx.x * a.slabs * kMmaCtaRows, r_end = min(a.R, r_first + a.slabs * kMmaCtaRows);
  // All of the CTA's weights are asked for in the L2 at once: the loads below hold no more in flight than a block of 256
  // values a lane.
  if (tid == 0) {
    prefetch_weight_rows<QT>(w[0], nblk, K, r_first, r_end);
    if constexpr (NMAT == 2) prefetch_weight_rows<QT>(w[1], nblk, K, r_first, r_end);
  }
  // The rows. Those past n are never written and their columns never stored.
  const uint32_t stride = K + mma_pad(QT), sum_stride = SL ? K / (SL ? SL : 1) + 8 : 0;
  float *scales = (float *)(smem + 8 * NT * stride);
  int16_t *sums = (int16_t *)(scales + 8 * NT * per_row);
  for (uint32_t i = tid; i < n * (K / 16); i += 256) {
    const uint32_t t = i / (K / 16), c = i % (K / 16);
    const uint64_t row = a.act_row ? a.act_row[start + t] : start + t;
    *(int4 *)(smem + t * stride + 16 * c) = ((const int4 *)(a.act.q + row * a.act.q_stride))[c];
  }
  for (uint32_t i = tid; i < n * per_row; i += 256) {
    const uint32_t t = i / per_row, c = i % per_row;
    const uint64_t row = a.act_row ? a.act_row[start + t] : start + t;
    scales[c * 8 * NT + t] = ((const float *)((const uint8_t *)a.act.d + row * a.act.d_stride))[c];
  }
  if constexpr (SL > 0)
    for (uint32_t i = tid; i < n * (K / SL); i += 256) {
      const uint32_t t = i / (K / SL), c = i % (K / SL);
      const uint64_t row = a.act_row ? a.act_row[start + t] : start + t;
      const int16_t *bs = (const int16_t *)((const uint8_t *)a.act.bs + row * a.act.bs_stride);
      sums[t * sum_stride + c] = SL == 16 ? bs[c] : (int16_t)(bs[2 * c] + bs[2 * c + 1]);
    }
  uint32_t *grid = (uint32_t *)(sums + 8 * NT * sum_stride);
  if constexpr (grid_words(QT) > 0)
    for (uint32_t i = tid; i < grid_words(QT); i += 256) grid[i] = __ldg(a.grid + grid_offset(QT) + i);
  __syncthreads();
  const MmaActs acts{smem, scales, sums, stride, sum_stride, grid};
  using F = Frag<QT>;
  for (uint32_t r0 = r_first + 16 * warp; r0 < r_end; r0 += kMmaCtaRows) {
    float f[NMAT][NT][4];
#pragma unroll
    for (int m = 0; m < NMAT; m++) {
#pragma unroll
      for (int t = 0; t < NT; t++) f[m][t][0] = f[m][t][1] = f[m][t][2] = f[m][t][3] = 0.0f;
      if constexpr (mma_ahead(QT)) {
        typename F::Row x = F::fetch(w[m], nblk, K, r0 + g, 0, j), y = F::fetch(w[m], nblk, K, r0 + g + 8, 0, j);
        for (uint32_t b = 0; b < KB; b++) {
          const typename F::Row cx = x, cy = y;
          if (b + 1 < KB) x = F::fetch(w[m], nblk, K, r0 + g, b + 1, j), y = F::fetch(w[m], nblk, K, r0 + g + 8, b + 1, j);
          F::template block<NT>(cx, cy, b, g, j, acts, f[m]);
        }
      } else {
        for (uint32_t b = 0; b < KB; b++) {
          const typename F::Row x = F::fetch(w[m], nblk, K, r0 + g, b, j), y = F::fetch(w[m], nblk, K, r0 + g + 8, b, j);
          F::template block<NT>(x, y, b, g, j, acts, f[m]);
        }
      }
    }
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint32_t col = 8 * t + 2 * j + (k & 1), r = r0 + g + (k & 2 ? 8 : 0);
        if (col >= n) continue;
        float v = f[0][t][k];
        if constexpr (NMAT == 2) v = swiglu(v, f[1][t][k], a.limit);
        const uint64_t o = (uint64_t)(start + col) * a.out_stride + r;
        if (a.out_f16)
          ((__half *)a.out)[o] = __float2half_rn(v);
        else
          ((float *)a.out)[o] = v;
      }
  }
}

// NMAT 2: h[row][r] = swiglu(gate_r . x, up_r . x); NMAT 1: y[row][r] = down_r . h. Launch: grid (R / (kMmaCtaRows * slabs),
// CTAs that share the entries), 256 threads, dynamic shared memory mma_smem(QT, 8 * MOST, K). MOST: tiles of 8 activation rows an entry
// may fill; one with fewer takes the form for as many as it has.
template <int QT, int NMAT, int MOST>
__global__ void __launch_bounds__(256, mma_ahead(QT) || MOST > 1 ? 2 : 3) k_expert_mma(const ExpertMmaArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  dependents_may_launch(), wait_for_predecessors();
  const uint32_t first = a.end ? *a.first : 0, n1 = a.end ? *a.end - first : 0, n2 = a.end2 ? *a.end2 : 0;
  for (uint32_t i = blockIdx.y; i < n1 + n2; i += gridDim.y) {
    const MoeGroup en = i < n1 ? a.entries[first + i] : a.entries2[i - n1];
    if (i != blockIdx.y) __syncthreads();  // the entry before has been read out of shared memory
    if constexpr (MOST == 1) {
      mma_entry<QT, NMAT, 1>(a, en, smem);
    } else {
      static_assert(MOST == 4, "as many forms as are called here");
      switch ((en.n + 7) / 8) {
        case 1: mma_entry<QT, NMAT, 1>(a, en, smem); break;
        case 2: mma_entry<QT, NMAT, 2>(a, en, smem); break;
        case 3: mma_entry<QT, NMAT, 3>(a, en, smem); break;
        default: mma_entry<QT, NMAT, 4>(a, en, smem);
      }
    }
  }
}

}  // namespace moe

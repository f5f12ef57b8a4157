// The experts' products for a few rows per expert (up to 32), exact as the integer-dot kernels are: the weights' codes as
// int8 against the rows' int8 codes on the warp-level tensor instruction (mma.sync, int8 in, int32 out), 16 weight rows
// by 8 activation rows an instruction, one sub-block of the weights (32 values, or 16 where the type scales 16) at
// a time; the integer sums then meet the sub-block's scale in int32 and the block's in f32, as the CPU path's dots do
// (core/cpu/experts.cpp:152-284).
//
// Why this unit and not tcgen05: its sums would leave tensor memory once per sub-block to be scaled, so the tile kernel
// decodes to f16 with the scales folded in, some 5.5 instructions a weight, and with a dozen rows an expert that decode is
// the whole of its time. Here a weight stays the code it is: for Q4_K an AND (and a shift) a word of eight, and some 3.5
// instructions a weight with 15 rows, multiply-adds, scales and all. The rows' codes are read from shared memory at one word
// per lane a sub-block, where dp4a needs a 16-byte piece per lane and row. What bounds it: with few rows HBM (Q8_0, 100 rows of
// the benchmark's layer: gate and up 167 us, 5.9 TB/s of weights; down 81 us, 6.0), with more the instructions (Q4_K, 777 rows: gate
// and up 191 us, issue slots two thirds busy).
//
// A warp takes 16 weight rows at a time over the whole row length. The blocks come through a ring of its own in shared memory,
// filled by 16-byte asynchronous copies whose lanes take neighbouring pieces of a row, and running on across the items the CTA
// takes one after another; which of a sub-block's values sit in which lane is free as long as both operands agree, and is
// chosen so that a lane's share of a sub-block is contiguous in memory. (Blocks loaded straight to registers, a block ahead, 32 bytes
// of eight rows a load: eight lines an instruction for the L1, whose data pipe then stood at 85 % while an SM had work, and
// a wait for memory at every item's start: the four launches above took 218, 111, 251 and 132 us.)
#pragma once

#include <type_traits>

#include "expert_rows.cuh"

namespace moe {

constexpr uint32_t kMmaRows = 32;               // activation rows an entry holds at most
constexpr uint32_t kMmaRowsUnit = 256;          // weight rows come in multiples of what a CTA of 16 warps takes at a time, 16 a warp
constexpr uint32_t kMmaMaxSmem = 100 * 1024;    // for the rows of an entry

// The rows in shared memory: codes with a stride that spreads eight rows' words over the banks; the scales, sub-block or
// block by block with the rows side by side; the sums of each 32 or 16 codes. Before them a codebook type's codebook and the warps' rings.
__host__ __device__ constexpr uint32_t mma_pad(uint32_t qt) { return qt == QT_Q6_K ? 16 : 32; }
__host__ __device__ constexpr uint32_t mma_sum_len(uint32_t qt) { return qt == QT_Q4_K ? 32 : qt == QT_Q6_K ? 16 : 0; }
__host__ __device__ constexpr uint32_t mma_smem(uint32_t qt, uint32_t rows, uint32_t K) {
  const uint32_t sums = mma_sum_len(qt) ? K / mma_sum_len(qt) * 2 + 16 : 0;
  return rows * (K + mma_pad(qt)) + rows * (act_is_q8k(qt) ? K / 256 : K / 32) * 4 + rows * sums + 4 * grid_words(qt);
}
// Whether the kernel takes entries of up to `rows` rows (8 or kMmaRows) of K values: a CTA holds them all.
__host__ __device__ constexpr bool mma_takes(uint32_t qt, uint32_t K, uint32_t rows) {
  return K % 256 == 0 && mma_smem(qt, rows, K) <= kMmaMaxSmem;
}

// Stages of a warp's ring: an entry of up to eight rows leaves room for four, in the types of whose blocks nothing is loaded to
// registers beside the ring.
__host__ __device__ constexpr uint32_t mma_stages(uint32_t qt, int most) {
  return most == 1 && (qt == QT_Q8_0 || qt == QT_Q4_K || qt == QT_IQ4_NL || qt == QT_Q2_0) ? 4 : 2;
}

struct ExpertMmaArgs {
  const uint8_t *w0, *w1;   // slot 0's slice of (gate, up) or (down, unused), runs layout
  uint64_t slice_bytes;
  uint32_t K, R;            // values per weight row; weight rows (a multiple of kMmaRowsUnit)
  ActView act;
  const uint32_t *act_row;  // expert-order row -> activation row; null: the same row
  const MoeGroup *entries;  // (slot, start, n), n <= kMmaRows: the list's entries *first .. *end
  const uint32_t *first, *end;
  const MoeGroup *entries2; // after them, entries 0 .. *end2 of a second list; either list may be left out (end null)
  const uint32_t *end2;
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
template <int BYTES>
__device__ __forceinline__ void cp_async_small(uint32_t dst_smem, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst_smem), "l"(src), "n"(BYTES) : "memory");
}

// A stage of a warp's ring: a block of 16 weight rows, field by field. SWIZZLE says which of a row's 16-byte pieces is stored
// where, so that the reads below fall on different banks: as it stands; pieces of 32 bytes by the row's low two bits (reads of 8
// bytes, four lanes to 32); pieces of 16 bytes by the row's place among those that the same read takes (reads of four lanes to
// one piece). It is an exclusive-or on the address, which a stage's and its fields' alignment to 128 bytes leaves room for, and
// the same for rows g and g + 8.
enum StageSwizzle { SW_NONE, SW_PAIRS, SW_PIECES };
template <uint32_t ROW, int SWIZZLE>
__device__ __forceinline__ uint32_t stage_swizzle(uint32_t row) {
  if constexpr (SWIZZLE == SW_PAIRS) return (row & 3) << 5;
  if constexpr (SWIZZLE == SW_PIECES) return row / (128 / ROW) % (ROW / 16) * 16;
  return 0;
}
// Byte `at` of the row, where its lane's reads start from: byte 16 c + at of the row is then at this ^ 16 c.
template <uint32_t ROW, int SWIZZLE>
__device__ __forceinline__ uint32_t stage_row(uint32_t field, uint32_t row, uint32_t at) {
  return field + ROW * row + stage_swizzle<ROW, SWIZZLE>(row) + at;
}
// ROW bytes of each of 16 rows into dst, `step` bytes from a row to the next at src.
template <uint32_t ROW, int SWIZZLE = SW_NONE>
__device__ __forceinline__ void stage_rows(uint32_t dst, const uint8_t *src, uint32_t step, uint32_t lane) {
  if constexpr (ROW < 16) {
    if (lane < 16) cp_async_small<ROW>(dst + ROW * lane, src + (uint64_t)lane * step);
  } else {
    constexpr uint32_t C = ROW / 16;  // pieces a row
#pragma unroll
    for (uint32_t i = 0; i < (C + 1) / 2; i++) {
      const uint32_t row = lane / C + i * (32 / C), c = lane % C;
      if (C > 1 || lane < 16) cp_async16(dst + ROW * row + (16 * c ^ stage_swizzle<ROW, SWIZZLE>(row)), src + (uint64_t)row * step + 16 * c);
    }
  }
}
struct NoSmall {};
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
// Byte i of w, signed: one permute, whose selector's fourth bits spread the byte's own sign.
__device__ __forceinline__ int sbyte(uint32_t w, int i) {
  int d;
  asm("prmt.b32 %0, %1, 0, %2;" : "=r"(d) : "r"(w), "r"(0x1110 * (8 + i) + i));
  return d;
}

// What a block's product reads of the rows: codes of row n at codes + n * stride; scales, NT * 8 rows side by side; sums of
// row n at sums + n * sum_stride (int16).
struct MmaActs {
  const uint8_t *codes;
  const float *scales;
  const int16_t *sums;
  uint32_t stride, sum_stride;
  const uint32_t *grid;  // a codebook type's codebook
};

// A type's share of a lane. A stage is kValues values of each of the warp's 16 rows, kStage bytes; issue() asks for one, Row is
// what a lane takes of one row's part of it (lane j = lane % 4 of the four that share the row). Small: what is no multiple of
// four bytes a row, loaded straight to registers a stage ahead. block() adds the products of two weight rows (g and g + 8 of the warp's 16, g = lane / 4) with columns
// 2 j, 2 j + 1 of each of the NT tiles of 8 activation rows to f.
template <int QT>
struct Frag;

// Q4_K: y = d * sc * q - dmin * m. A pair of sub-blocks is 32 bytes, their low and high nibbles; a lane's share 8 of them:
// values 8 j .. 8 j + 7 of either sub-block.
template <>
struct Frag<QT_Q4_K> {
  static constexpr uint32_t kValues = 256, kStage = 16 * 144;
  using Small = NoSmall;
  struct Row {
    uint2 q[4];
    uint4 hd;
  };
  __device__ static __forceinline__ void issue(uint32_t dst, const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r0, uint32_t b, uint32_t lane) {
    const uint64_t blk = (uint64_t)r0 * (K / 256) + b;
    stage_rows<128, SW_PAIRS>(dst, s + 128 * blk, K / 2, lane);
    stage_rows<16>(dst + 2048, s + 128 * nblk + 16 * blk, K / 16, lane);
  }
  __device__ static __forceinline__ Row load(const uint8_t *smem, uint32_t st, uint32_t row, uint32_t j, const Small &) {
    Row x;
#pragma unroll
    for (int p = 0; p < 4; p++) x.q[p] = *(const uint2 *)(smem + (stage_row<128, SW_PAIRS>(st, row, 8 * j) ^ 32 * p));
    x.hd = *(const uint4 *)(smem + st + 2048 + 16 * row);
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
  static constexpr uint32_t kValues = 128, kStage = 16 * 136;
  using Small = NoSmall;
  struct Row {
    uint2 q[4], d;
  };
  __device__ static __forceinline__ void issue(uint32_t dst, const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r0, uint32_t b, uint32_t lane) {
    stage_rows<128, SW_PAIRS>(dst, s + (uint64_t)r0 * K + 128 * b, K, lane);
    stage_rows<8>(dst + 2048, s + 32 * nblk + (uint64_t)r0 * (K / 16) + 8 * b, K / 16, lane);
  }
  __device__ static __forceinline__ Row load(const uint8_t *smem, uint32_t st, uint32_t row, uint32_t j, const Small &) {
    Row x;
#pragma unroll
    for (int i = 0; i < 4; i++) x.q[i] = *(const uint2 *)(smem + (stage_row<128, SW_PAIRS>(st, row, 8 * j) ^ 32 * i));
    x.d = *(const uint2 *)(smem + st + 2048 + 8 * row);
    return x;
  }
  __device__ static __forceinline__ float half_of(uint32_t w, int i) {
    const __half2 h = *(const __half2 *)&w;
    return i & 1 ? __high2float(h) : __low2float(h);
  }
  template <int NT>
  __device__ static __forceinline__ void block(const Row &x, const Row &y, uint32_t b, uint32_t g, uint32_t j, const MmaActs &acts, float (&f)[NT][4]) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float dx = half_of(i < 2 ? x.d.x : x.d.y, i), dy = half_of(i < 2 ? y.d.x : y.d.y, i);
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const uint2 v = *(const uint2 *)(acts.codes + (8 * t + g) * acts.stride + 128 * b + 32 * i + 8 * j);
        const float2 da = *(const float2 *)(acts.scales + (4 * b + i) * 8 * NT + 8 * t + 2 * j);
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
  static constexpr uint32_t kValues = 256, kStage = 16 * 208;
  using Small = __half;  // d
  struct Row {
    uint32_t l[8], h[4];
    uint4 sc;
    float d;
  };
  __device__ static __forceinline__ void issue(uint32_t dst, const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r0, uint32_t b, uint32_t lane) {
    const uint64_t blk = (uint64_t)r0 * (K / 256) + b;
    stage_rows<128, SW_PIECES>(dst, s + 128 * blk, K / 2, lane);
    stage_rows<64, SW_PIECES>(dst + 2048, s + 128 * nblk + 64 * blk, K / 4, lane);
    stage_rows<16>(dst + 3072, s + 192 * nblk + 16 * blk, K / 16, lane);
  }
  __device__ static __forceinline__ Small small(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t b) {
    return __ldg((const __half *)(s + 208 * nblk) + (uint64_t)r * (K / 256) + b);
  }
  __device__ static __forceinline__ Row load(const uint8_t *smem, uint32_t st, uint32_t row, uint32_t j, const Small &d) {
    Row x;
#pragma unroll
    for (int i = 0; i < 8; i++) x.l[i] = *(const uint32_t *)(smem + (stage_row<128, SW_PIECES>(st, row, 4 * j) ^ 16 * i));
#pragma unroll
    for (int i = 0; i < 4; i++) x.h[i] = *(const uint32_t *)(smem + (stage_row<64, SW_PIECES>(st + 2048, row, 4 * j) ^ 16 * i));
    x.sc = *(const uint4 *)(smem + st + 3072 + 16 * row);
    x.d = __half2float(d);
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
// lane's share is four bytes, looked up in the order their nibbles have (values v, 16 + v, v + 1, 17 + v of a word): the rows' codes
// are staged in that order too (mma_stage_acts), so nothing parts low nibbles from high ones.
__host__ __device__ constexpr bool mma_paired(uint32_t qt) { return qt == QT_IQ4_XS || qt == QT_IQ4_NL; }
// y = d * (ls - 32) * table[q], a 6-bit ls a sub-block.
template <>
struct Frag<QT_IQ4_XS> {
  static constexpr uint32_t kValues = 256, kStage = 2048 + 128;
  struct Small {
    uint16_t sh;
    __half d;
  };
  struct Row {
    uint32_t q[8], sl, sh;
    float d;
  };
  __device__ static __forceinline__ void issue(uint32_t dst, const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r0, uint32_t b, uint32_t lane) {
    const uint64_t blk = (uint64_t)r0 * (K / 256) + b;
    stage_rows<128, SW_PIECES>(dst, s + 128 * blk, K / 2, lane);
    stage_rows<4>(dst + 2048, s + 128 * nblk + 4 * blk, K / 64, lane);
  }
  __device__ static __forceinline__ Small small(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t b) {
    const uint64_t blk = (uint64_t)r * (K / 256) + b;
    return Small{__ldg((const uint16_t *)(s + 132 * nblk) + blk), __ldg((const __half *)(s + 134 * nblk) + blk)};
  }
  __device__ static __forceinline__ Row load(const uint8_t *smem, uint32_t st, uint32_t row, uint32_t j, const Small &o) {
    Row x;
#pragma unroll
    for (int i = 0; i < 8; i++) x.q[i] = *(const uint32_t *)(smem + (stage_row<128, SW_PIECES>(st, row, 4 * j) ^ 16 * i));
    x.sl = *(const uint32_t *)(smem + st + 2048 + 4 * row), x.sh = o.sh, x.d = __half2float(o.d);
    return x;
  }
  template <int NT>
  __device__ static __forceinline__ void block(const Row &x, const Row &y, uint32_t b, uint32_t g, uint32_t j, const MmaActs &acts, float (&f)[NT][4]) {
    int sum[NT][4];
#pragma unroll
    for (int t = 0; t < NT; t++) sum[t][0] = sum[t][1] = sum[t][2] = sum[t][3] = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint2 ax = iq4_pairs<0>(x.q[i]), ay = iq4_pairs<0>(y.q[i]);
      const int sx = (int)(((x.sl >> (4 * i)) & 0xF) | (((x.sh >> (2 * i)) & 3) << 4)) - 32, sy = (int)(((y.sl >> (4 * i)) & 0xF) | (((y.sh >> (2 * i)) & 3) << 4)) - 32;
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const uint2 v = *(const uint2 *)(acts.codes + (8 * t + g) * acts.stride + 256 * b + 32 * i + 8 * j);
        int c[4];
        mma_k32(c, ax.x, ay.x, ax.y, ay.y, v.x, v.y);
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
  static constexpr uint32_t kValues = 256, kStage = 16 * 144;
  using Small = NoSmall;
  struct Row {
    uint32_t q[8];
    uint4 d;
  };
  __device__ static __forceinline__ void issue(uint32_t dst, const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r0, uint32_t b, uint32_t lane) {
    stage_rows<128, SW_PIECES>(dst, s + (uint64_t)r0 * (K / 2) + 128 * b, K / 2, lane);
    stage_rows<16>(dst + 2048, s + 16 * nblk + (uint64_t)r0 * (K / 16) + 16 * b, K / 16, lane);
  }
  __device__ static __forceinline__ Row load(const uint8_t *smem, uint32_t st, uint32_t row, uint32_t j, const Small &) {
    Row x;
#pragma unroll
    for (int i = 0; i < 8; i++) x.q[i] = *(const uint32_t *)(smem + (stage_row<128, SW_PIECES>(st, row, 4 * j) ^ 16 * i));
    x.d = *(const uint4 *)(smem + st + 2048 + 16 * row);
    return x;
  }
  __device__ static __forceinline__ float scale(const uint4 &d, int i) {
    return Frag<QT_Q8_0>::half_of(i < 2 ? d.x : i < 4 ? d.y : i < 6 ? d.z : d.w, i);
  }
  template <int NT>
  __device__ static __forceinline__ void block(const Row &x, const Row &y, uint32_t b, uint32_t g, uint32_t j, const MmaActs &acts, float (&f)[NT][4]) {
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint2 ax = iq4_pairs<0>(x.q[i]), ay = iq4_pairs<0>(y.q[i]);
      const float dx = scale(x.d, i), dy = scale(y.d, i);
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const float2 da = *(const float2 *)(acts.scales + (8 * b + i) * 8 * NT + 8 * t + 2 * j);
        const uint2 v = *(const uint2 *)(acts.codes + (8 * t + g) * acts.stride + 256 * b + 32 * i + 8 * j);
        int c[4];
        mma_k32(c, ax.x, ay.x, ax.y, ay.y, v.x, v.y);
        f[t][0] = fmaf(dx * da.x, (float)c[0], f[t][0]), f[t][1] = fmaf(dx * da.y, (float)c[1], f[t][1]);
        f[t][2] = fmaf(dy * da.x, (float)c[2], f[t][2]), f[t][3] = fmaf(dy * da.y, (float)c[3], f[t][3]);
      }
    }
  }
};

// The two bytes that are a lane's share of sub-block i in a run of 64 bytes a row, from the lane's place in the row.
__device__ __forceinline__ uint32_t quad_share(const uint8_t *smem, uint32_t at, int i) {
  return *(const uint16_t *)(smem + (at ^ 16 * (i / 2)) + 8 * (i & 1));
}
__device__ __forceinline__ uint32_t byte_of(const uint2 &v, int i) { return ((i < 4 ? v.x : v.y) >> (8 * (i & 3))) & 0xFF; }
// Word w with the bits `mask` of v, moved so that v's bit `from` comes to bit `to`.
__device__ __forceinline__ uint32_t bits_at(uint32_t w, uint32_t v, int from, int to, uint32_t mask) {
  return w | ((from >= to ? v >> (from - to) : v << (to - from)) & mask);
}

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
  static constexpr uint32_t kValues = 256, kStage = 1664 + 128;
  using Small = __half;  // d
  struct Row {
    const uint8_t *smem;
    uint32_t qs, sg;         // the lane's places in the stage
    uint2 qh;                // shifted to the lane's two bits of each byte
    uint32_t sc;
    float d;
  };
  __device__ static __forceinline__ void issue(uint32_t dst, const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r0, uint32_t b, uint32_t lane) {
    const uint64_t blk = (uint64_t)r0 * (K / 256) + b;
    stage_rows<64, SW_PIECES>(dst, s + 64 * blk, K / 4, lane);
    stage_rows<32, SW_PIECES>(dst + 1024, s + 64 * nblk + 32 * blk, K / 8, lane);
    stage_rows<8>(dst + 1536, s + 96 * nblk + 8 * blk, K / 32, lane);
    stage_rows<4>(dst + 1664, s + 104 * nblk + 4 * blk, K / 64, lane);
  }
  __device__ static __forceinline__ Small small(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t b) {
    return __ldg((const __half *)(s + 108 * nblk) + (uint64_t)r * (K / 256) + b);
  }
  __device__ static __forceinline__ Row load(const uint8_t *smem, uint32_t st, uint32_t row, uint32_t j, const Small &d) {
    Row x;
    x.smem = smem, x.qs = stage_row<64, SW_PIECES>(st, row, 2 * j), x.sg = stage_row<32, SW_PIECES>(st + 1024, row, j);
    const uint2 qh = *(const uint2 *)(smem + st + 1536 + 8 * row);
    x.qh = make_uint2(qh.x >> (2 * j), qh.y >> (2 * j));
    x.sc = *(const uint32_t *)(smem + st + 1664 + 4 * row), x.d = __half2float(d);
    return x;
  }
  __device__ static __forceinline__ void words(const Row &x, int i, uint32_t, const uint32_t *grid, uint32_t (&a)[2]) {
    const uint32_t q = quad_share(x.smem, x.qs, i), h = i < 4 ? x.qh.x : x.qh.y, sb = x.smem[(x.sg ^ 16 * (i / 4)) + 4 * (i & 3)];
    a[0] = (uint32_t)signed_word(grid[bits_at(q & 0xFF, h, 8 * (i & 3), 8, 0x100u)], sb & 0xF);
    a[1] = (uint32_t)signed_word(grid[bits_at(q >> 8, h, 8 * (i & 3) + 1, 8, 0x100u)], sb >> 4);
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
  static constexpr uint32_t kValues = 256, kStage = 16 * 96;
  using Small = __half;  // d
  struct Row {
    const uint8_t *smem;
    uint32_t qs;  // the lane's place in the stage
    uint4 w[2];
    float d;
  };
  __device__ static __forceinline__ void issue(uint32_t dst, const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r0, uint32_t b, uint32_t lane) {
    const uint64_t blk = (uint64_t)r0 * (K / 256) + b;
    stage_rows<64, SW_PIECES>(dst, s + 64 * blk, K / 4, lane);
    stage_rows<32, SW_PIECES>(dst + 1024, s + 64 * nblk + 32 * blk, K / 8, lane);
  }
  __device__ static __forceinline__ Small small(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t b) {
    return __ldg((const __half *)(s + 96 * nblk) + (uint64_t)r * (K / 256) + b);
  }
  __device__ static __forceinline__ Row load(const uint8_t *smem, uint32_t st, uint32_t row, uint32_t j, const Small &d) {
    Row x;
    x.smem = smem, x.qs = stage_row<64, SW_PIECES>(st, row, 2 * j);
#pragma unroll
    for (int c = 0; c < 2; c++) x.w[c] = *(const uint4 *)(smem + (stage_row<32, SW_PIECES>(st + 1024, row, 0) ^ 16 * c));
    x.d = 0.25f * __half2float(d);  // (2 s + 1) / 4 = (0.5 + s) / 2
    return x;
  }
  __device__ static __forceinline__ void words(const Row &x, int i, uint32_t j, const uint32_t *grid, uint32_t (&a)[2]) {
    const uint32_t q = quad_share(x.smem, x.qs, i), k7 = (word_of(x.w, i) >> (7 * j)) & 127u, sb = k7 | ((__popc(k7) & 1u) << 7);
    a[0] = (uint32_t)signed_word(grid[q & 0xFF], sb & 0xF), a[1] = (uint32_t)signed_word(grid[q >> 8], sb >> 4);
  }
  __device__ static __forceinline__ uint32_t word_of(const uint4 (&v)[2], int i) {
    const uint4 &u = v[i / 4];
    return (i & 3) == 0 ? u.x : (i & 3) == 1 ? u.y : (i & 3) == 2 ? u.z : u.w;
  }
  __device__ static __forceinline__ int scale(const Row &x, int i) { return 2 * (int)(word_of(x.w, i) >> 28) + 1; }
  template <int NT>
  __device__ static __forceinline__ void block(const Row &x, const Row &y, uint32_t b, uint32_t g, uint32_t j, const MmaActs &acts, float (&f)[NT][4]) {
    block_of_words<Frag, NT>(x, y, b, g, j, acts, f);
  }
};

// IQ2_S: y = d * (0.5 + s) / 4 * grid[index][i] * sign, a 10-bit index and a byte of signs for each eight values, an s for
// each 16. A lane's share of a sub-block of 32 is one entry, both its words, so that an index is put together once for eight
// values (an instruction for each 16 values, whose lanes take half an entry, put it together twice: 73 experts' gate and up
// 87 us, at the rate of the ALU pipe). The sub-block's two scales then meet its two halves' sums: the first half's by
// an instruction whose activations of the other half, lanes 2 and 3, are zero; the second's is the rest.
template <>
struct Frag<QT_IQ2_S> {
  static constexpr uint32_t kValues = 256, kStage = 16 * 80;
  using Small = __half;  // d
  struct Row {
    const uint8_t *smem;
    uint32_t qs, sg;         // the lane's places in the stage
    uint2 qh, sc;            // qh shifted to the lane's two bits of each byte
    float d;
  };
  __device__ static __forceinline__ void issue(uint32_t dst, const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r0, uint32_t b, uint32_t lane) {
    const uint64_t blk = (uint64_t)r0 * (K / 256) + b;
    stage_rows<32, SW_PIECES>(dst, s + 32 * blk, K / 8, lane);
    stage_rows<32, SW_PIECES>(dst + 512, s + 32 * nblk + 32 * blk, K / 8, lane);
    stage_rows<8>(dst + 1024, s + 64 * nblk + 8 * blk, K / 32, lane);
    stage_rows<8>(dst + 1152, s + 72 * nblk + 8 * blk, K / 32, lane);
  }
  __device__ static __forceinline__ Small small(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t b) {
    return __ldg((const __half *)(s + 80 * nblk) + (uint64_t)r * (K / 256) + b);
  }
  __device__ static __forceinline__ Row load(const uint8_t *smem, uint32_t st, uint32_t row, uint32_t j, const Small &d) {
    Row x;
    x.smem = smem, x.qs = stage_row<32, SW_PIECES>(st, row, j), x.sg = x.qs + 512;
    const uint2 qh = *(const uint2 *)(smem + st + 1024 + 8 * row);
    x.qh = make_uint2(qh.x >> (2 * j), qh.y >> (2 * j)), x.sc = *(const uint2 *)(smem + st + 1152 + 8 * row);
    x.d = 0.125f * __half2float(d);  // (2 s + 1) / 8 = (0.5 + s) / 4
    return x;
  }
  __device__ static __forceinline__ void words(const Row &x, int i, const uint32_t *grid, uint32_t (&a)[2]) {
    const uint32_t sb = x.smem[(x.sg ^ 16 * (i / 4)) + 4 * (i & 3)];
    const uint2 e = ((const uint2 *)grid)[bits_at(x.smem[(x.qs ^ 16 * (i / 4)) + 4 * (i & 3)], i < 4 ? x.qh.x : x.qh.y, 8 * (i & 3), 8, 0x300u)];
    a[0] = (uint32_t)signed_word(e.x, sb & 0xF), a[1] = (uint32_t)signed_word(e.y, sb >> 4);
  }
  template <int NT>
  __device__ static __forceinline__ void block(const Row &x, const Row &y, uint32_t b, uint32_t g, uint32_t j, const MmaActs &acts, float (&f)[NT][4]) {
    int sum[NT][4];
#pragma unroll
    for (int t = 0; t < NT; t++) sum[t][0] = sum[t][1] = sum[t][2] = sum[t][3] = 0;
    const uint32_t first_half = j < 2 ? 0xFFFFFFFFu : 0u;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      uint32_t ax[2], ay[2];
      words(x, i, acts.grid, ax), words(y, i, acts.grid, ay);
      // 2 s + 1 of the second half, and how much more the first half's is: sum = s1 * all + (s0 - s1) * first.
      const uint32_t scx = byte_of(x.sc, i), scy = byte_of(y.sc, i);
      const int sx = 2 * (int)(scx >> 4) + 1, sy = 2 * (int)(scy >> 4) + 1, dx = 2 * (int)(scx & 0xF) + 1 - sx, dy = 2 * (int)(scy & 0xF) + 1 - sy;
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const uint2 v = *(const uint2 *)(acts.codes + (8 * t + g) * acts.stride + 256 * b + 32 * i + 8 * j);
        int c[4], h[4];
        mma_k32(c, ax[0], ay[0], ax[1], ay[1], v.x, v.y);
        mma_k32(h, ax[0], ay[0], ax[1], ay[1], v.x & first_half, v.y & first_half);
        sum[t][0] += sx * c[0] + dx * h[0], sum[t][1] += sx * c[1] + dx * h[1], sum[t][2] += sy * c[2] + dy * h[2], sum[t][3] += sy * c[3] + dy * h[3];
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
  static constexpr uint32_t kValues = 256, kStage = 16 * 72;
  using Small = NoSmall;
  struct Row {
    const uint8_t *smem;
    uint32_t q;  // the lane's place in the stage
    uint2 d;
  };
  __device__ static __forceinline__ void issue(uint32_t dst, const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r0, uint32_t b, uint32_t lane) {
    stage_rows<64, SW_PIECES>(dst, s + (uint64_t)r0 * (K / 4) + 64 * b, K / 4, lane);
    stage_rows<8>(dst + 1024, s + 16 * nblk + (uint64_t)r0 * (K / 32) + 8 * b, K / 32, lane);
  }
  __device__ static __forceinline__ Row load(const uint8_t *smem, uint32_t st, uint32_t row, uint32_t j, const Small &) {
    Row x;
    x.smem = smem, x.q = stage_row<64, SW_PIECES>(st, row, 2 * j), x.d = *(const uint2 *)(smem + st + 1024 + 8 * row);
    return x;
  }
  // Two bytes of four codes each, q - 1 as signed bytes: the codes spread to the digits of two permutes' selectors.
  __device__ static __forceinline__ void q2_words(uint32_t q, uint32_t &lo, uint32_t &hi) {
    uint32_t u = __byte_perm(q, 0, 0x4140u);
    u = (u | u << 4) & 0x0F0F0F0Fu, u = (u | u << 2) & 0x33333333u;
    lo = __byte_perm(0x020100FFu, 0u, u), hi = __byte_perm(0x020100FFu, 0u, u >> 16);
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
      uint32_t a0, a1, a2, a3;
      q2_words(quad_share(x.smem, x.q, i), a0, a2), q2_words(quad_share(y.smem, y.q, i), a1, a3);
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

// The rows of an entry into shared memory, for NT tiles of 8 columns. Those past n are never written and their columns never stored.
template <int QT>
__device__ __forceinline__ MmaActs mma_stage_acts(const ExpertMmaArgs &a, const MoeGroup &en, uint32_t NT, uint8_t *smem, const uint32_t *grid) {
  constexpr uint32_t SL = mma_sum_len(QT);
  const uint32_t K = a.K, n = en.n, start = en.start, per_row = act_is_q8k(QT) ? K / 256 : K / 32;
  const uint32_t stride = K + mma_pad(QT), sum_stride = SL ? K / (SL ? SL : 1) + 8 : 0;
  float *scales = (float *)(smem + 8 * NT * stride);
  int16_t *sums = (int16_t *)(scales + 8 * NT * per_row);
  if constexpr (mma_paired(QT)) {
    for (uint32_t i = threadIdx.x; i < n * (K / 32); i += blockDim.x) {
      const uint32_t t = i / (K / 32), c = i % (K / 32);
      const uint64_t row = a.act_row ? a.act_row[start + t] : start + t;
      const uint4 lo = ((const uint4 *)(a.act.q + row * a.act.q_stride))[2 * c], hi = ((const uint4 *)(a.act.q + row * a.act.q_stride))[2 * c + 1];
      uint4 *dst = (uint4 *)(smem + t * stride + 32 * c);
      dst[0] = make_uint4(__byte_perm(lo.x, hi.x, 0x5140u), __byte_perm(lo.x, hi.x, 0x7362u), __byte_perm(lo.y, hi.y, 0x5140u), __byte_perm(lo.y, hi.y, 0x7362u));
      dst[1] = make_uint4(__byte_perm(lo.z, hi.z, 0x5140u), __byte_perm(lo.z, hi.z, 0x7362u), __byte_perm(lo.w, hi.w, 0x5140u), __byte_perm(lo.w, hi.w, 0x7362u));
    }
  } else {
    for (uint32_t i = threadIdx.x; i < n * (K / 16); i += blockDim.x) {
      const uint32_t t = i / (K / 16), c = i % (K / 16);
      const uint64_t row = a.act_row ? a.act_row[start + t] : start + t;
      *(int4 *)(smem + t * stride + 16 * c) = ((const int4 *)(a.act.q + row * a.act.q_stride))[c];
    }
  }
  for (uint32_t i = threadIdx.x; i < n * per_row; i += blockDim.x) {
    const uint32_t t = i / per_row, c = i % per_row;
    const uint64_t row = a.act_row ? a.act_row[start + t] : start + t;
    scales[c * 8 * NT + t] = ((const float *)((const uint8_t *)a.act.d + row * a.act.d_stride))[c];
  }
  if constexpr (SL > 0)
    for (uint32_t i = threadIdx.x; i < n * (K / SL); i += blockDim.x) {
      const uint32_t t = i / (K / SL), c = i % (K / SL);
      const uint64_t row = a.act_row ? a.act_row[start + t] : start + t;
      const int16_t *bs = (const int16_t *)((const uint8_t *)a.act.bs + row * a.act.bs_stride);
      sums[t * sum_stride + c] = SL == 16 ? bs[c] : (int16_t)(bs[2 * c] + bs[2 * c + 1]);
    }
  return MmaActs{smem, scales, sums, stride, sum_stride, grid};
}

// What a warp asks for ahead of what it multiplies: its items one after another, of each the matrices, of each the stages.
struct MmaAhead {
  uint32_t k = 0, m = 0, b = 0;          // the item in the CTA's order, the matrix, the stage
  uint32_t entry = 0xFFFFFFFFu, r0 = 0;  // the item's entry and the warp's rows
  uint64_t slice = 0;
  uint32_t slot = 0;                     // of the ring
};

// NMAT 2: h[row][r] = swiglu(gate_r . x, up_r . x); NMAT 1: y[row][r] = down_r . h. An item is 16 weight rows a warp of an entry.
// Launch: a round of CTAs or a few, or as many as the lists can hold items; 8 or 16 warps; dynamic shared memory the warps'
// rings and mma_smem(QT, 8 * MOST, K). How many entries there are the lists on the device say: the CTAs take an item each or,
// where there are more, two runs of consecutive ones, one from the front of the order and its mirror image from the end, for
// the short tiles are listed by falling row count. An entry's rows are staged once for a run's items, and the rings run on from
// one to the next. MOST: tiles of 8 activation rows an entry may fill; one with fewer takes the form for as many as it has.
__host__ __device__ constexpr int mma_threads(int most) { return most == 1 ? 256 : 512; }
template <int QT, int NMAT, int MOST>
__global__ void __launch_bounds__(mma_threads(MOST), MOST > 1 ? 1 : grid_words(QT) ? 3 : 2) k_expert_mma(const ExpertMmaArgs a) {
  extern __shared__ __align__(128) uint8_t smem[];
  dependents_may_launch(), wait_for_predecessors();
  using F = Frag<QT>;
  static_assert(F::kStage % 128 == 0, "stage_row");
  using Small = typename F::Small;
  constexpr uint32_t S = mma_stages(QT, MOST);
  constexpr bool kSmall = !std::is_same<Small, NoSmall>::value;
  static_assert(!kSmall || S == 2, "what is loaded to registers is a stage ahead");
  const uint32_t first = a.end ? *a.first : 0, n1 = a.end ? *a.end - first : 0, n2 = a.end2 ? *a.end2 : 0;
  const uint32_t K = a.K, KB = K / F::kValues, warps = blockDim.x / 32, slab = 16 * warps, per_entry = a.R / slab;
  const uint64_t nblk = (uint64_t)a.R * (K / block_values(QT));
  const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32, g = lane / 4, j = lane % 4;
  auto entry_at = [&](uint32_t e) { return e < n1 ? a.entries[first + e] : a.entries2[e - n1]; };
  // The CTA's items: len0 from from0 on, then those from from1 on. CTAs past the items leave.
  const uint64_t items = (uint64_t)(n1 + n2) * per_entry;
  const uint32_t ctas = (uint32_t)min((uint64_t)gridDim.x, items), c = blockIdx.x;
  if (c >= ctas) return;
  auto cut = [&](uint32_t k) { return (uint32_t)(k * items / (2 * ctas)); };
  const uint32_t from0 = cut(c), len0 = cut(c + 1) - from0, from1 = cut(2 * ctas - 1 - c), len = len0 + cut(2 * ctas - c) - from1;
  auto item_at = [&](uint32_t k) { return k < len0 ? from0 + k : from1 + (k - len0); };

  uint32_t *grid = (uint32_t *)smem;
  const uint32_t ring = 4 * grid_words(QT) + warp * (S * F::kStage), ring32 = (uint32_t)__cvta_generic_to_shared(smem) + ring;
  uint8_t *rows = smem + 4 * grid_words(QT) + warps * (S * F::kStage);
  MmaAhead ah;
  Small next_x{}, next_y{};
  auto ask = [&]() {
    if (ah.k < len) {
      if (ah.m == 0 && ah.b == 0) {
        const uint32_t item = item_at(ah.k), e = item / per_entry;
        if (e != ah.entry) ah.entry = e, ah.slice = entry_at(e).slot * a.slice_bytes;
        ah.r0 = (item % per_entry) * slab + 16 * warp;
      }
      const uint8_t *w = (NMAT == 2 && ah.m ? a.w1 : a.w0) + ah.slice;
      F::issue(ring32 + ah.slot * F::kStage, w, nblk, K, ah.r0, ah.b, lane);
      if constexpr (kSmall) next_x = F::small(w, nblk, K, ah.r0 + g, ah.b), next_y = F::small(w, nblk, K, ah.r0 + g + 8, ah.b);
      ah.slot = ah.slot + 1 == S ? 0 : ah.slot + 1;
      if (++ah.b == KB) {
        ah.b = 0;
        if (++ah.m == NMAT) ah.m = 0, ah.k++;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (uint32_t i = 0; i + 1 < S; i++) ask();
  if constexpr (grid_words(QT) > 0)
    for (uint32_t i = threadIdx.x; i < grid_words(QT); i += blockDim.x) grid[i] = __ldg(a.grid + grid_offset(QT) + i);

  uint32_t staged = 0xFFFFFFFFu, slot = 0;
  MoeGroup en{};
  MmaActs acts{};
  auto take = [&](auto tiles, uint32_t r0) {
    constexpr int NT = decltype(tiles)::value;
    float f[NMAT][NT][4];
#pragma unroll
    for (int m = 0; m < NMAT; m++) {
#pragma unroll
      for (int t = 0; t < NT; t++) f[m][t][0] = f[m][t][1] = f[m][t][2] = f[m][t][3] = 0.0f;
      for (uint32_t b = 0; b < KB; b++) {
        [[maybe_unused]] const Small sx = next_x, sy = next_y;
        __syncwarp();  // every lane has read the stage that is asked for again now
        ask();
        asm volatile("cp.async.wait_group %0;" ::"n"(S - 1) : "memory");
        __syncwarp();
        const uint32_t st = ring + slot * F::kStage;
        slot = slot + 1 == S ? 0 : slot + 1;
        const typename F::Row x = F::load(smem, st, g, j, sx), y = F::load(smem, st, g + 8, j, sy);
        F::template block<NT>(x, y, b, g, j, acts, f[m]);
      }
    }
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint32_t col = 8 * t + 2 * j + (k & 1), r = r0 + g + (k & 2 ? 8 : 0);
        if (col >= en.n) continue;
        float v = f[0][t][k];
        if constexpr (NMAT == 2) v = swiglu(v, f[1][t][k], a.limit);
        const uint64_t o = (uint64_t)(en.start + col) * a.out_stride + r;
        if (a.out_f16)
          ((__half *)a.out)[o] = __float2half_rn(v);
        else
          ((float *)a.out)[o] = v;
      }
  };
  for (uint32_t k = 0; k < len; k++) {
    const uint32_t item = item_at(k), e = item / per_entry;
    if (e != staged) {
      if (staged != 0xFFFFFFFFu) __syncthreads();  // the entry before has been read out of shared memory
      en = entry_at(e), staged = e;
      acts = mma_stage_acts<QT>(a, en, MOST == 1 ? 1 : (en.n + 7) / 8, rows, grid);
      __syncthreads();
    }
    const uint32_t r0 = (item % per_entry) * slab + 16 * warp;
    if constexpr (MOST == 1) {
      take(std::integral_constant<int, 1>{}, r0);
    } else {
      static_assert(MOST == 4, "as many forms as are called here");
      switch ((en.n + 7) / 8) {
        case 1: take(std::integral_constant<int, 1>{}, r0); break;
        case 2: take(std::integral_constant<int, 2>{}, r0); break;
        case 3: take(std::integral_constant<int, 3>{}, r0); break;
        default: take(std::integral_constant<int, 4>{}, r0);
      }
    }
  }
}

}  // namespace moe

// The experts' products for few rows per expert: integer dots of quantised weights against int8 activations, a group
// of lanes per weight row, 128-bit loads of the quants in the runs layout, the weights decoded once in registers for
// every row of the group, shuffle reductions. This is the bandwidth-bound path (decode and draft-verify steps); it
// replaces the reference's grouped GEMVs (kernels/quant/moe.cl:230-302,416-471; kernels/quant/matvec.cl:101-159) and
// follows the arithmetic of its CPU path (core/cpu/experts.cpp:152-284): activations as q8_0 or q8_K, integer block
// sums, f32 scales.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "cuda_rt.h"
#include "formats.h"
#include "iq4nl_values.h"
#include "quant_rows.cuh"
#include "router_topk.cuh"

namespace moe {

// One expert's rows start .. start + count of the expert order, at most kTileRows of them.
struct MoeTile {
  uint32_t expert, slot, start, count;
};
// Rows start .. start + n of the expert order, all of one expert (its slot among this GPU's experts), n <= 8: the
// reference's MoeGroup (shared/moe_tile.h:20-33) with the rows named by their place in expert order.
struct MoeGroup {
  uint32_t slot, start, n;
};
constexpr int kGroupMax = 8;

// Quantised activation rows: a row's K codes at q + row * q_stride; its scales at d + row * d_stride bytes (q8_0: K/32
// floats, the f16 scale widened; q8_K: K/256 floats); q8_K's sums of each 16 codes at bs + row * bs_stride bytes. The
// strides let the three parts be arrays of their own or pieces of one packed row.
struct ActView {
  const int8_t *q;
  const float *d;
  const int16_t *bs;
  uint32_t q_stride, d_stride, bs_stride;
};

// A step that takes the short form (forward_short): at most so many rows, and assignments of rows to experts.
constexpr uint32_t kShortRows = 8, kShortMax = 64;

// Rows start .. start + count of the expert order, all of one expert; count <= kTileN.
struct BigTile {
  uint32_t slot, start, count;
};

// Which experts with one short tile go to the few-rows kernel: none; those of up to 16 rows, or 32 in a step that hits many
// experts; all of them if none has more than 8, else none.
enum FewRows { FEW_NONE, FEW_BY_ROWS, FEW_IF_ALL };

// What a pack leaves: the step's assignments by expert, and the lists the experts' kernels walk.
struct PackOut {
  uint32_t *cnt, *base;    // NE each
  uint32_t *chunk_off;     // [chunks][NE]: rows of the expert's run taken by earlier chunks
  MoeTile *tiles;          // expert order, <= 64 rows each (prompt.cl:719-723)
  MoeGroup *groups;        // <= group_max rows each: the experts with fewer than tensor_min rows
  BigTile *big;            // <= kTileN rows each: the others, for the tensor-core kernels
  uint32_t *counters;      // [0] tiles, [1] groups, [2] experts hit, [3] rows, [4] big tiles, [5] their rows, [6] the first of the
                           // big tiles that go to the few-rows kernel (expert_mma.cuh): short ones, at the list's end
  uint32_t few_rows;       // how the scan settles which (FewRows)
};

// A short step's route: exact logits in; ids, weights, gates and the lists out, those of at most kShortMax assignments by
// comparing each with every other, where k_router_topk_pack scans all the experts through 1,024 threads.
struct ShortRoute {
  const float *rl;      // [T][NE + 1], exact
  uint32_t T, NE, K;    // K experts a row
  uint32_t group_max;   // rows a listed group holds
  int32_t *ids;
  float *w, *gs;
  uint32_t *inv, *row_src;
  PackOut o;            // chunk_off is not written
};
struct ExpertRowsArgs {
  const uint8_t *w0, *w1;  // slot 0's slice of the matrix (gate, up) or (down, unused), runs layout
  uint64_t slice_bytes;    // from one slot's slice to the next
  uint32_t K, R;           // values per weight row; weight rows
  uint32_t rows_per_cta;
  ActView act;
  const uint32_t *act_row;  // expert-order row -> activation row; null: the same row
  const MoeGroup *groups;   // null: dense_rows rows of slot 0, taken M at a time
  const uint32_t *ngroups;
  uint32_t dense_rows;
  uint32_t halves;          // CTAs, along the grid's third extent, that share a group M rows each (0 or 1: one takes it whole)
  uint32_t slabs;           // row slabs a CTA takes one after another (0 or 1: one); only with the row length known at compile time
  float *out;  // out[expert-order row][r]
  uint32_t out_stride;
  float limit;  // SwiGLU limit, 0: off
  const float *act_f32;  // QUANT: the activation rows before quantisation, [rows][K]; act and act_row are not read
  ShortRoute route;      // ROUTED: act_row, groups and ngroups are not read
  QuantJob codes;        // QUANT: where the quantised rows are left too (q null: nowhere)
};

__device__ __forceinline__ uint4 ldg_stream16(const void *p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
// `bytes` from p on (both multiples of 16) asked for in the L2.
__device__ __forceinline__ void prefetch_l2_bulk(const void *p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ int dot4x4(const uint4 &w, const int4 &a) {
  int s = __dp4a((int)w.x, a.x, 0);
  s = __dp4a((int)w.y, a.y, s);
  s = __dp4a((int)w.z, a.z, s);
  return __dp4a((int)w.w, a.w, s);
}

// Bytes of one activation row in shared memory: codes, then the scales (padded to 16), then q8_K's sums.
__host__ __device__ constexpr uint32_t act_d_bytes(bool q8k, uint32_t K) { return q8k ? ((K / 64 + 15) & ~15u) : K / 8; }
constexpr uint32_t kRowsMaxK = 16384;  // the longest activation row the integer-dot kernels stage (8 rows of it fit an SM's shared memory)
// Row lengths that the integer-dot kernels have forms of their own for (launch_shape): the benchmark's, and a row of one block.
constexpr uint32_t kRowsLengths[] = {2048, 512, 256};
constexpr bool rows_specialised(uint32_t K) {
  for (uint32_t n : kRowsLengths)
    if (n == K) return true;
  return false;
}
__host__ __device__ constexpr uint32_t act_row_stride(bool q8k, uint32_t K) { return K + act_d_bytes(q8k, K) + (q8k ? K / 8 : 0) + 16; }

// SwiGLU as the CPU path states it (core/cpu/experts.cpp:21-27).
__device__ __forceinline__ float swiglu(float g, float u, float limit) {
  if (limit > 0.0f) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
  }
  return g / (1.0f + expf(-g)) * u;
}

// One lane's unit of a weight row: what it loads (Raw, 16 bytes of quants and the scales beside them) and its dot with
// the matching codes of M activation rows. nblk: blocks in the slice; r: row; u: unit within the row.
template <int QT>
struct Unit;

// Q8_0: y = d * q (docs/spec/QUANT_FORMATS.md:461). A unit is 16 codes, half a block.
template <>
struct Unit<QT_Q8_0> {
  static constexpr int kValues = 16;
  struct Raw {
    uint4 q;
    float d;
  };
  __device__ static __forceinline__ Raw fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t u, const uint32_t *) {
    Raw x;
    x.q = ldg_stream16(s + (uint64_t)r * K + 16u * u);
    x.d = __half2float(__ldg((const __half *)(s + 32 * nblk) + (uint64_t)r * (K / 32) + u / 2));
    return x;
  }
  template <int M>
  __device__ static __forceinline__ void dot(const Raw &x, uint32_t K, uint32_t u, const uint8_t *acts, uint32_t stride, float *acc, uint32_t n) {
#pragma unroll
    for (int t = 0; t < M; t++) {
      if ((uint32_t)t >= n) break;  // the group's rows: the same for the whole CTA
      const uint8_t *a = acts + t * stride;
      const int s = dot4x4(x.q, *(const int4 *)(a + 16u * u));
      acc[t] = fmaf(x.d * ((const float *)(a + K))[u / 2], (float)s, acc[t]);
    }
  }
};

// Q4_K: y = d * sc * q - dmin * m, eight sub-blocks of 32 with 6-bit sc and m (QUANT_FORMATS.md:373-394). A unit is
// 16 bytes of qs: 16 values of sub-block 2p in the low nibbles, 16 of sub-block 2p + 1 in the high ones.
template <>
struct Unit<QT_Q4_K> {
  static constexpr int kValues = 32;
  struct Raw {
    uint4 q;
    uint32_t s0, s1, s2;
    __half2 dm;
  };
  __device__ static __forceinline__ Raw fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t u, const uint32_t *) {
    Raw x;
    x.q = ldg_stream16(s + (uint64_t)r * (K / 2) + 16u * u);
    const uint64_t blk = (uint64_t)r * (K / 256) + u / 8;
    const uint4 hd = __ldg((const uint4 *)(s + 128 * nblk + 16 * blk));  // d, dmin, then the 12 bytes of scales
    x.dm = *(const __half2 *)&hd.x;
    x.s0 = hd.y, x.s1 = hd.z, x.s2 = hd.w;
    return x;
  }
  __device__ static __forceinline__ uint32_t byte_of(const Raw &x, int i) {
    const uint32_t w = i < 4 ? x.s0 : i < 8 ? x.s1 : x.s2;
    return (w >> (8 * (i & 3))) & 0xFF;
  }
  // The packed scale and minimum of sub-block j (QUANT_FORMATS.md:386-392).
  __device__ static __forceinline__ void scale_min(const Raw &x, int j, int &sc, int &m) {
    if (j < 4) {
      sc = byte_of(x, j) & 63;
      m = byte_of(x, j + 4) & 63;
    } else {
      sc = (byte_of(x, j + 4) & 0xF) | ((byte_of(x, j - 4) >> 6) << 4);
      m = (byte_of(x, j + 4) >> 4) | ((byte_of(x, j) >> 6) << 4);
    }
  }
  template <int M>
  __device__ static __forceinline__ void dot(const Raw &x, uint32_t K, uint32_t u, const uint8_t *acts, uint32_t stride, float *acc, uint32_t n) {
    const uint32_t b = u / 8, j = u % 8, p = j / 2, hf = j & 1;
    int sc_lo, m_lo, sc_hi, m_hi;
    scale_min(x, 2 * p, sc_lo, m_lo);
    scale_min(x, 2 * p + 1, sc_hi, m_hi);
    const uint4 lo = make_uint4(x.q.x & 0x0F0F0F0Fu, x.q.y & 0x0F0F0F0Fu, x.q.z & 0x0F0F0F0Fu, x.q.w & 0x0F0F0F0Fu);
    const uint4 hi = make_uint4((x.q.x >> 4) & 0x0F0F0F0Fu, (x.q.y >> 4) & 0x0F0F0F0Fu, (x.q.z >> 4) & 0x0F0F0F0Fu,
                                (x.q.w >> 4) & 0x0F0F0F0Fu);
    const float d = __low2float(x.dm), dmin = __high2float(x.dm);
    const uint32_t dsz = act_d_bytes(true, K);
#pragma unroll
    for (int t = 0; t < M; t++) {
      if ((uint32_t)t >= n) break;  // the group's rows: the same for the whole CTA
      const uint8_t *a = acts + t * stride;
      const uint8_t *av = a + 256 * b + 64 * p + 16 * hf;
      const int s_lo = dot4x4(lo, *(const int4 *)av), s_hi = dot4x4(hi, *(const int4 *)(av + 32));
      const int16_t *bs = (const int16_t *)(a + K + dsz) + 16 * b + 4 * p + hf;
      const float da = ((const float *)(a + K))[b];
      acc[t] += da * (d * (float)(sc_lo * s_lo + sc_hi * s_hi) - dmin * (float)(m_lo * bs[0] + m_hi * bs[2]));
    }
  }
};

// Q6_K: y = d * scales[v / 16] * (q - 32), 6-bit codes split into ql (low 4) and qh (high 2) (QUANT_FORMATS.md:419-441).
// A unit is 16 bytes of ql with the 16 bytes of qh that complete them: 16 values in the low nibbles and 16 in the high
// ones, each a whole group of 16 with its own int8 scale.
template <>
struct Unit<QT_Q6_K> {
  static constexpr int kValues = 32;
  struct Raw {
    uint4 ql, qh;
    int sc_lo, sc_hi;
    float d;
  };
  __device__ static __forceinline__ Raw fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t u, const uint32_t *) {
    Raw x;
    x.ql = ldg_stream16(s + (uint64_t)r * (K / 2) + 16u * u);
    const uint32_t j = u % 8, h = j / 4, jj = j % 4;
    const uint64_t blk = (uint64_t)r * (K / 256) + u / 8;
    x.qh = ldg_stream16(s + 128 * nblk + 64 * blk + 32 * h + 16 * (jj & 1));
    const int8_t *sc = (const int8_t *)(s + 192 * nblk + 16 * blk) + 8 * h + 2 * (jj >> 1) + (jj & 1);
    x.sc_lo = __ldg(sc), x.sc_hi = __ldg(sc + 4);
    x.d = __half2float(__ldg((const __half *)(s + 208 * nblk) + blk));
    return x;
  }
  template <int M>
  __device__ static __forceinline__ void dot(const Raw &x, uint32_t K, uint32_t u, const uint8_t *acts, uint32_t stride, float *acc, uint32_t n) {
    const uint32_t b = u / 8, j = u % 8, h = j / 4, jj = j % 4, sh = jj < 2 ? 0 : 2;
    const uint32_t g16 = 8 * h + 2 * (jj >> 1) + (jj & 1);  // the low nibbles' group of 16; the high ones' is 4 on
    uint4 lo, hi;
    lo.x = (x.ql.x & 0x0F0F0F0Fu) | (((x.qh.x >> sh) & 0x03030303u) << 4);
    lo.y = (x.ql.y & 0x0F0F0F0Fu) | (((x.qh.y >> sh) & 0x03030303u) << 4);
    lo.z = (x.ql.z & 0x0F0F0F0Fu) | (((x.qh.z >> sh) & 0x03030303u) << 4);
    lo.w = (x.ql.w & 0x0F0F0F0Fu) | (((x.qh.w >> sh) & 0x03030303u) << 4);
    hi.x = ((x.ql.x >> 4) & 0x0F0F0F0Fu) | (((x.qh.x >> (sh + 4)) & 0x03030303u) << 4);
    hi.y = ((x.ql.y >> 4) & 0x0F0F0F0Fu) | (((x.qh.y >> (sh + 4)) & 0x03030303u) << 4);
    hi.z = ((x.ql.z >> 4) & 0x0F0F0F0Fu) | (((x.qh.z >> (sh + 4)) & 0x03030303u) << 4);
    hi.w = ((x.ql.w >> 4) & 0x0F0F0F0Fu) | (((x.qh.w >> (sh + 4)) & 0x03030303u) << 4);
    const uint32_t dsz = act_d_bytes(true, K);
#pragma unroll
    for (int t = 0; t < M; t++) {
      if ((uint32_t)t >= n) break;  // the group's rows: the same for the whole CTA
      const uint8_t *a = acts + t * stride;
      const uint8_t *av = a + 256 * b + 16 * g16;
      const int s_lo = dot4x4(lo, *(const int4 *)av), s_hi = dot4x4(hi, *(const int4 *)(av + 64));
      const int16_t *bs = (const int16_t *)(a + K + dsz) + 16 * b + g16;
      const int isum = x.sc_lo * (s_lo - 32 * bs[0]) + x.sc_hi * (s_hi - 32 * bs[4]);
      acc[t] = fmaf(x.d * ((const float *)(a + K))[b], (float)isum, acc[t]);
    }
  }
};

// IQ3_S: y = d * (1 + 2 s) * grid[index][i] * sign, 9-bit indices into the 512-entry codebook, one per 4 values
// (QUANT_FORMATS.md:178-207). A unit is 16 bytes of qs: two sub-blocks of 32. The codebook sits in shared memory; the
// signs go onto the codebook's bytes once, for every activation row.
template <>
struct Unit<QT_IQ3_S> {
  static constexpr int kValues = 64;
  struct Raw {
    uint4 qs;
    uint2 sg;
    uint32_t qh, sc;
    float d;
  };
  __device__ static __forceinline__ Raw fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t u, const uint32_t *) {
    Raw x;
    x.qs = ldg_stream16(s + (uint64_t)r * (K / 4) + 16u * u);
    const uint32_t c = u % 4;
    const uint64_t blk = (uint64_t)r * (K / 256) + u / 4;
    x.sg = __ldg((const uint2 *)(s + 64 * nblk + 32 * blk + 8 * c));
    x.qh = __ldg((const uint16_t *)(s + 96 * nblk + 8 * blk + 2 * c));
    x.sc = __ldg(s + 104 * nblk + 4 * blk + c);
    x.d = __half2float(__ldg((const __half *)(s + 108 * nblk) + blk));
    return x;
  }
  template <int M>
  __device__ static __forceinline__ void dot(const Raw &x, uint32_t K, uint32_t u, const uint8_t *acts, uint32_t stride, float *acc,
                                             uint32_t n, const uint32_t *grid) {
    const uint32_t b = u / 4, c = u % 4;
    // A codebook word is four values in 1 .. 15; a sign bit negates its byte: (v ^ 0xFF) + 1 = 256 - v stays within the
    // byte for v >= 1, so the four bytes take one exclusive-or and one 32-bit add. The nibble's bits reach the bytes'
    // low bits by one multiply: bit i times 2^(7 i) lands on bit 8 i, and no two products share a bit.
    int g[16];
    const uint32_t qh9 = x.qh << 8;
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const uint32_t word = i < 4 ? x.qs.x : i < 8 ? x.qs.y : i < 12 ? x.qs.z : x.qs.w;
      const uint32_t idx = ((word >> (8 * (i & 3))) & 0xFF) | ((qh9 >> i) & 0x100u);
      const uint32_t nib = ((i < 8 ? x.sg.x : x.sg.y) >> (4 * (i & 7))) & 0xF;
      const uint32_t lsb = (nib * 0x00204081u) & 0x01010101u;
      g[i] = (int)((grid[idx] ^ (lsb * 0xFFu)) + lsb);
    }
    const int sc0 = 2 * (int)(x.sc & 0xF) + 1, sc1 = 2 * (int)((x.sc >> 4) & 0xF) + 1;
#pragma unroll
    for (int t = 0; t < M; t++) {
      if ((uint32_t)t >= n) break;  // the group's rows: the same for the whole CTA
      const uint8_t *a = acts + t * stride;
      const int4 *av = (const int4 *)(a + 256 * b + 64 * c);
      const uint32_t sw = (u >> 1) & 3;  // act_slot's swizzle
      const int4 a0 = av[0 ^ sw], a1 = av[1 ^ sw], a2 = av[2 ^ sw], a3 = av[3 ^ sw];
      int s0 = __dp4a(g[0], a0.x, 0), s1 = __dp4a(g[8], a2.x, 0);
      s0 = __dp4a(g[1], a0.y, s0), s1 = __dp4a(g[9], a2.y, s1);
      s0 = __dp4a(g[2], a0.z, s0), s1 = __dp4a(g[10], a2.z, s1);
      s0 = __dp4a(g[3], a0.w, s0), s1 = __dp4a(g[11], a2.w, s1);
      s0 = __dp4a(g[4], a1.x, s0), s1 = __dp4a(g[12], a3.x, s1);
      s0 = __dp4a(g[5], a1.y, s0), s1 = __dp4a(g[13], a3.y, s1);
      s0 = __dp4a(g[6], a1.z, s0), s1 = __dp4a(g[14], a3.z, s1);
      s0 = __dp4a(g[7], a1.w, s0), s1 = __dp4a(g[15], a3.w, s1);
      acc[t] = fmaf(x.d * ((const float *)(a + K))[b], (float)(sc0 * s0 + sc1 * s1), acc[t]);
    }
  }
};

// A codebook word's four bytes made negative where the nibble's bits say so. A byte is in 1 .. 127, so (v ^ 0xFF) + 1 =
// 256 - v stays within the byte and the four take one exclusive-or and one 32-bit add; the nibble's bits reach the
// bytes' low bits by one multiply: bit i times 2^(7 i) lands on bit 8 i, and no two products share a bit.
__device__ __forceinline__ int signed_word(uint32_t g, uint32_t nib) {
  const uint32_t lsb = (nib * 0x00204081u) & 0x01010101u;
  return (int)((g ^ (lsb * 0xFFu)) + lsb);
}
// 8 activation words of a sub-block against 8 decoded words.
__device__ __forceinline__ int dot8(const int *g, const int4 &a0, const int4 &a1) {
  int s = __dp4a(g[0], a0.x, 0);
  s = __dp4a(g[1], a0.y, s), s = __dp4a(g[2], a0.z, s), s = __dp4a(g[3], a0.w, s);
  s = __dp4a(g[4], a1.x, s), s = __dp4a(g[5], a1.y, s), s = __dp4a(g[6], a1.z, s), s = __dp4a(g[7], a1.w, s);
  return s;
}

// IQ3_XXS: y = d * (0.5 + s) / 2 * grid[index][i] * sign: 8-bit indices into a 256-entry codebook, one per 4 values;
// a sub-block of 32 has one word: four 7-bit sign indices (the eighth sign of each 8 values is the index's parity)
// and the 4-bit s (QUANT_FORMATS.md:147-173). A unit is 16 bytes of indices: two sub-blocks.
template <>
struct Unit<QT_IQ3_XXS> {
  static constexpr int kValues = 64;
  struct Raw {
    uint4 qs;
    uint2 gas;
    float d;
  };
  __device__ static __forceinline__ Raw fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t u, const uint32_t *) {
    Raw x;
    x.qs = ldg_stream16(s + (uint64_t)r * (K / 4) + 16u * u);
    const uint32_t c = u % 4;
    const uint64_t blk = (uint64_t)r * (K / 256) + u / 4;
    x.gas = __ldg((const uint2 *)(s + 64 * nblk + 32 * blk + 8 * c));
    x.d = 0.25f * __half2float(__ldg((const __half *)(s + 96 * nblk) + blk));  // (2 s + 1) / 4 = (0.5 + s) / 2
    return x;
  }
  template <int M>
  __device__ static __forceinline__ void dot(const Raw &x, uint32_t K, uint32_t u, const uint8_t *acts, uint32_t stride, float *acc,
                                             uint32_t n, const uint32_t *grid) {
    const uint32_t b = u / 4, c = u % 4;
    int g[16];
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const uint32_t word = i < 4 ? x.qs.x : i < 8 ? x.qs.y : i < 12 ? x.qs.z : x.qs.w;
      const uint32_t w32 = i < 8 ? x.gas.x : x.gas.y;
      const uint32_t k7 = (w32 >> (7 * ((i & 7) >> 1))) & 127u, sbyte = k7 | ((__popc(k7) & 1u) << 7);
      g[i] = signed_word(grid[(word >> (8 * (i & 3))) & 0xFF], (sbyte >> (4 * (i & 1))) & 0xF);
    }
    const int sc0 = 2 * (int)(x.gas.x >> 28) + 1, sc1 = 2 * (int)(x.gas.y >> 28) + 1;
#pragma unroll
    for (int t = 0; t < M; t++) {
      if ((uint32_t)t >= n) break;  // the group's rows: the same for the whole CTA
      const uint8_t *a = acts + t * stride;
      const int4 *av = (const int4 *)(a + 256 * b + 64 * c);
      const uint32_t sw = (u >> 1) & 3;  // act_slot's swizzle
      const int s0 = dot8(g, av[0 ^ sw], av[1 ^ sw]), s1 = dot8(g + 8, av[2 ^ sw], av[3 ^ sw]);
      acc[t] = fmaf(x.d * ((const float *)(a + K))[b], (float)(sc0 * s0 + sc1 * s1), acc[t]);
    }
  }
};

// IQ2_S: y = d * (0.5 + s) / 4 * grid[index][i] * sign: 10-bit indices into a 1024-entry codebook of 8 values (8 bits in
// qs, 2 in qh), a byte of signs a group, a 4-bit s per 16 values (QUANT_FORMATS.md:115-145). A unit is 8 bytes of qs:
// two sub-blocks of 32. The codebook in shared memory is two words an entry.
template <>
struct Unit<QT_IQ2_S> {
  static constexpr int kValues = 64;
  struct Raw {
    uint2 qs, sg;
    uint32_t qh, sc;
    float d;
  };
  __device__ static __forceinline__ Raw fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t u, const uint32_t *) {
    Raw x;
    x.qs = __ldg((const uint2 *)(s + (uint64_t)r * (K / 8) + 8u * u));
    const uint32_t c = u % 4;
    const uint64_t blk = (uint64_t)r * (K / 256) + u / 4;
    x.sg = __ldg((const uint2 *)(s + 32 * nblk + 32 * blk + 8 * c));
    x.qh = __ldg((const uint16_t *)(s + 64 * nblk + 8 * blk + 2 * c));
    x.sc = __ldg((const uint16_t *)(s + 72 * nblk + 8 * blk + 2 * c));
    x.d = 0.125f * __half2float(__ldg((const __half *)(s + 80 * nblk) + blk));  // (2 s + 1) / 8 = (0.5 + s) / 4
    return x;
  }
  template <int M>
  __device__ static __forceinline__ void dot(const Raw &x, uint32_t K, uint32_t u, const uint8_t *acts, uint32_t stride, float *acc,
                                             uint32_t n, const uint32_t *grid) {
    const uint32_t b = u / 4, c = u % 4;
    const uint2 *grid2 = (const uint2 *)grid;
    int g[16];
#pragma unroll
    for (int j = 0; j < 8; j++) {  // group j: sub-block j / 4, its group j % 4
      const uint32_t lo8 = ((j < 4 ? x.qs.x : x.qs.y) >> (8 * (j & 3))) & 0xFF;
      const uint32_t hi2 = ((x.qh >> (8 * (j >> 2))) >> (2 * (j & 3))) & 3u;
      const uint32_t sb = ((j < 4 ? x.sg.x : x.sg.y) >> (8 * (j & 3))) & 0xFF;
      const uint2 e = grid2[lo8 | (hi2 << 8)];
      g[2 * j] = signed_word(e.x, sb & 0xF), g[2 * j + 1] = signed_word(e.y, sb >> 4);
    }
    // 2 s + 1 of the four 16-value halves.
    const int k0 = 2 * (int)(x.sc & 0xF) + 1, k1 = 2 * (int)((x.sc >> 4) & 0xF) + 1, k2 = 2 * (int)((x.sc >> 8) & 0xF) + 1,
              k3 = 2 * (int)((x.sc >> 12) & 0xF) + 1;
#pragma unroll
    for (int t = 0; t < M; t++) {
      if ((uint32_t)t >= n) break;  // the group's rows: the same for the whole CTA
      const uint8_t *a = acts + t * stride;
      const int4 *av = (const int4 *)(a + 256 * b + 64 * c);
      const uint32_t sw = (u >> 1) & 3;  // act_slot's swizzle
      const int4 a0 = av[0 ^ sw], a1 = av[1 ^ sw], a2 = av[2 ^ sw], a3 = av[3 ^ sw];
      int p0 = __dp4a(g[0], a0.x, 0), p1 = __dp4a(g[4], a1.x, 0), p2 = __dp4a(g[8], a2.x, 0), p3 = __dp4a(g[12], a3.x, 0);
      p0 = __dp4a(g[1], a0.y, p0), p1 = __dp4a(g[5], a1.y, p1), p2 = __dp4a(g[9], a2.y, p2), p3 = __dp4a(g[13], a3.y, p3);
      p0 = __dp4a(g[2], a0.z, p0), p1 = __dp4a(g[6], a1.z, p1), p2 = __dp4a(g[10], a2.z, p2), p3 = __dp4a(g[14], a3.z, p3);
      p0 = __dp4a(g[3], a0.w, p0), p1 = __dp4a(g[7], a1.w, p1), p2 = __dp4a(g[11], a2.w, p2), p3 = __dp4a(g[15], a3.w, p3);
      acc[t] = fmaf(x.d * ((const float *)(a + K))[b], (float)(k0 * p0 + k1 * p1 + k2 * p2 + k3 * p3), acc[t]);
    }
  }
};

// The 16-entry table of IQ4_NL and IQ4_XS as four words of four signed bytes, entries 4 i .. 4 i + 3 in word i.
__host__ __device__ constexpr uint32_t iq4_table_word(int i) {
  return (uint32_t)(uint8_t)kIq4nlValues[4 * i] | (uint32_t)(uint8_t)kIq4nlValues[4 * i + 1] << 8 | (uint32_t)(uint8_t)kIq4nlValues[4 * i + 2] << 16 |
         (uint32_t)(uint8_t)kIq4nlValues[4 * i + 3] << 24;
}
// Table values of the eight nibbles of q: lo = those of its four bytes' low nibbles (byte order kept), hi = of the
// high ones. A byte permute looks four nibbles up at once: its selector's digits are the nibbles' low three bits
// (entries 0 .. 7 from the table's first two words, 8 .. 15 from its last two), and a second permute takes each
// byte from the one or the other by the nibble's fourth bit. A third pair of permutes parts even nibbles from odd.
__device__ __forceinline__ void iq4_lookup8(uint32_t q, uint32_t &lo, uint32_t &hi) {
  constexpr uint32_t T0 = iq4_table_word(0), T1 = iq4_table_word(1), T2 = iq4_table_word(2), T3 = iq4_table_word(3);
  const uint32_t qa = q & 0xFFFFu, qb = q >> 16;
  const uint32_t sa = qa & 0x7777u, sb = qb & 0x7777u;
  const uint32_t r0 = __byte_perm(__byte_perm(T0, T1, sa), __byte_perm(T2, T3, sa), 0x3210u | ((qa & 0x8888u) >> 1));
  const uint32_t r1 = __byte_perm(__byte_perm(T0, T1, sb), __byte_perm(T2, T3, sb), 0x3210u | ((qb & 0x8888u) >> 1));
  lo = __byte_perm(r0, r1, 0x6420u), hi = __byte_perm(r0, r1, 0x7531u);
}

// Table values of q's eight nibbles in the order the nibbles have: .x those of its low two bytes (low nibble, high nibble, low,
// high), .y of its high two; each byte plus BIAS. Where both operands of a dot or a later permute agree on that order, the
// parting permutes of iq4_lookup8 are saved.
template <int BIAS>
__device__ __forceinline__ uint2 iq4_pairs(uint32_t q) {
  constexpr uint32_t B = 0x01010101u * BIAS;  // 0 or 128: the sign bits flipped
  constexpr uint32_t T0 = iq4_table_word(0) ^ B, T1 = iq4_table_word(1) ^ B, T2 = iq4_table_word(2) ^ B, T3 = iq4_table_word(3) ^ B;
  static_assert(BIAS == 0 || BIAS == 128, "an exclusive-or adds nothing else");
  const uint32_t e = q & 0x77777777u, half = (q >> 1 & 0x44444444u) | 0x32103210u;
  return make_uint2(__byte_perm(__byte_perm(T0, T1, e), __byte_perm(T2, T3, e), half),
                    __byte_perm(__byte_perm(T0, T1, e >> 16), __byte_perm(T2, T3, e >> 16), half >> 16));
}

// Sixteen 2-bit codes (a word's low or high half: 4 bytes of 4 codes) as 16 signed bytes q - 1 in four words. A byte's
// four codes are spread to the digits of a permute selector, whose table is the bytes -1, 0, 1, 2.
__device__ __forceinline__ uint32_t q2_bytes(uint32_t c) {  // c: one byte, four codes
  const uint32_t sel = (c & 0x3u) | ((c & 0xCu) << 2) | ((c & 0x30u) << 4) | ((c & 0xC0u) << 6);
  return __byte_perm(0x020100FFu, 0u, sel);
}

// Q2_0: y = (q - 1) * d, 64 values in 16 bytes with an f16 scale, value j in bits 2 (j mod 4) of byte j / 4
// (QUANT_FORMATS.md:251-270). A unit is one block; it meets two q8_0 blocks of activations, each with its own scale.
template <>
struct Unit<QT_Q2_0> {
  static constexpr int kValues = 64;
  struct Raw {
    uint4 q;
    float d;
  };
  __device__ static __forceinline__ Raw fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t u, const uint32_t *) {
    Raw x;
    x.q = ldg_stream16(s + (uint64_t)r * (K / 4) + 16u * u);
    x.d = __half2float(__ldg((const __half *)(s + 16 * nblk) + (uint64_t)r * (K / 64) + u));
    return x;
  }
  template <int M>
  __device__ static __forceinline__ void dot(const Raw &x, uint32_t K, uint32_t u, const uint8_t *acts, uint32_t stride, float *acc, uint32_t n) {
    int g[16];
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const uint32_t word = i < 4 ? x.q.x : i < 8 ? x.q.y : i < 12 ? x.q.z : x.q.w;
      g[i] = (int)q2_bytes((word >> (8 * (i & 3))) & 0xFF);
    }
#pragma unroll
    for (int t = 0; t < M; t++) {
      if ((uint32_t)t >= n) break;  // the group's rows: the same for the whole CTA
      const uint8_t *a = acts + t * stride;
      const int4 *av = (const int4 *)(a + 64u * u);
      const int s0 = dot8(g, av[0], av[1]), s1 = dot8(g + 8, av[2], av[3]);
      const float *da = (const float *)(a + K) + 2 * u;
      acc[t] = fmaf(x.d * da[0], (float)s0, acc[t]);
      acc[t] = fmaf(x.d * da[1], (float)s1, acc[t]);
    }
  }
};

// IQ4_NL: y = d * table[q], blocks of 32 with an f16 scale; a block's 16 bytes hold values 0 .. 15 in their low nibbles
// and 16 .. 31 in their high ones (QUANT_FORMATS.md:236-247). A unit is one block. Activations are q8_0.
template <>
struct Unit<QT_IQ4_NL> {
  static constexpr int kValues = 32;
  struct Raw {
    uint4 q;
    float d;
  };
  __device__ static __forceinline__ Raw fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t u, const uint32_t *) {
    Raw x;
    x.q = ldg_stream16(s + (uint64_t)r * (K / 2) + 16u * u);
    x.d = __half2float(__ldg((const __half *)(s + 16 * nblk) + (uint64_t)r * (K / 32) + u));
    return x;
  }
  template <int M>
  __device__ static __forceinline__ void dot(const Raw &x, uint32_t K, uint32_t u, const uint8_t *acts, uint32_t stride, float *acc, uint32_t n) {
    uint4 lo, hi;
    iq4_lookup8(x.q.x, lo.x, hi.x), iq4_lookup8(x.q.y, lo.y, hi.y), iq4_lookup8(x.q.z, lo.z, hi.z), iq4_lookup8(x.q.w, lo.w, hi.w);
#pragma unroll
    for (int t = 0; t < M; t++) {
      if ((uint32_t)t >= n) break;  // the group's rows: the same for the whole CTA
      const uint8_t *a = acts + t * stride;
      const int4 *av = (const int4 *)(a + 32u * u);
      const int s = dot4x4(lo, av[0]) + dot4x4(hi, av[1]);
      acc[t] = fmaf(x.d * ((const float *)(a + K))[u], (float)s, acc[t]);
    }
  }
};

// IQ4_XS: y = d * (ls - 32) * table[q], 256 values in eight sub-blocks of 32, each with a 6-bit ls: its low four bits
// a nibble of scales_l, its high two a pair of bits of scales_h (QUANT_FORMATS.md:213-232). A unit is one sub-block,
// 16 bytes of qs laid out as IQ4_NL's. Activations are q8_K (its sums are not needed: the table has no offset).
template <>
struct Unit<QT_IQ4_XS> {
  static constexpr int kValues = 32;
  struct Raw {
    uint4 q;
    uint32_t sl, sh;
    float d;
  };
  __device__ static __forceinline__ Raw fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t u, const uint32_t *) {
    Raw x;
    x.q = ldg_stream16(s + (uint64_t)r * (K / 2) + 16u * u);
    const uint64_t blk = (uint64_t)r * (K / 256) + u / 8;
    x.sl = __ldg((const uint32_t *)(s + 128 * nblk) + blk);
    x.sh = __ldg((const uint16_t *)(s + 132 * nblk) + blk);
    x.d = __half2float(__ldg((const __half *)(s + 134 * nblk) + blk));
    return x;
  }
  template <int M>
  __device__ static __forceinline__ void dot(const Raw &x, uint32_t K, uint32_t u, const uint8_t *acts, uint32_t stride, float *acc, uint32_t n) {
    const uint32_t b = u / 8, ib = u % 8;
    const int ls = (int)(((x.sl >> (4 * ib)) & 0xF) | (((x.sh >> (2 * ib)) & 3) << 4)) - 32;
    uint4 lo, hi;
    iq4_lookup8(x.q.x, lo.x, hi.x), iq4_lookup8(x.q.y, lo.y, hi.y), iq4_lookup8(x.q.z, lo.z, hi.z), iq4_lookup8(x.q.w, lo.w, hi.w);
#pragma unroll
    for (int t = 0; t < M; t++) {
      if ((uint32_t)t >= n) break;  // the group's rows: the same for the whole CTA
      const uint8_t *a = acts + t * stride;
      const int4 *av = (const int4 *)(a + 256 * b + 32 * ib);
      const int s = dot4x4(lo, av[0]) + dot4x4(hi, av[1]);
      acc[t] = fmaf(x.d * ((const float *)(a + K))[b], (float)(ls * s), acc[t]);
    }
  }
};

template <int QT, int M>
__device__ __forceinline__ void unit_dot(const typename Unit<QT>::Raw &x, uint32_t K, uint32_t u, const uint8_t *acts, uint32_t stride,
                                         float *acc, uint32_t n, const uint32_t *grid) {
  if constexpr (grid_words(QT) > 0)
    Unit<QT>::template dot<M>(x, K, u, acts, stride, acc, n, grid);
  else
    Unit<QT>::template dot<M>(x, K, u, acts, stride, acc, n);
}

// Where the 16-byte piece i of an activation row's codes sits in shared memory. The codebook types' units read four pieces 64 bytes
// apart from lane to lane, which without a swizzle puts a quarter-warp on two groups of four banks (four wavefronts an
// access instead of one): piece (i & 3) of unit i / 4 is stored at (i & 3) ^ ((unit >> 1) & 3).
template <int QT>
__device__ __forceinline__ uint32_t act_slot(uint32_t i) {
  if constexpr (grid_words(QT) > 0) return (i & ~3u) | ((i & 3u) ^ ((i >> 3) & 3u));
  return i;
}

// 16-byte loads a lane keeps in flight: with 8 the Q8_0 kernels fit three CTAs on an SM (16 took 114 registers, two CTAs),
// measured 2 to 5 % faster on steps of 1 to 32 rows.
constexpr int kRowsInFlight = 8;

// Passes of a warp whose loads are issued together: about kRowsInFlight loads of 16 bytes a lane, fewer when many activation rows
// already fill the registers with accumulators.
__host__ __device__ constexpr int rows_batch(int nmat, int nu, int m, bool heavy) {
  // heavy: a unit that holds many registers while it waits (IQ3_S: quants, signs, high bits, scale): fewer passes at
  // once leave room for more CTAs on the SM (three with one pass of gate and up, measured faster than two passes; two
  // passes for the down product, measured faster than one), which its arithmetic-bound decode needs more than loads
  // in flight.
  const int want = kRowsInFlight / (nmat * nu) > 0 ? kRowsInFlight / (nmat * nu) : 1, cap = heavy ? (nmat == 2 ? 1 : 2) : m >= 4 ? 4 : 8;
  return want < cap ? want : cap;
}

// Block blk of 256 values of a row, held eight a lane, quantised into the row's place in shared memory.
template <int QT>
__device__ __forceinline__ QuantLane stage_quantized(const float4 &v0, const float4 &v1, uint32_t blk, uint32_t lane, uint8_t *dst, uint32_t K) {
  constexpr bool q8k = act_is_q8k(QT);
  const QuantLane o = quantize_lane<q8k>(v0, v1, lane);
  *(uint2 *)(dst + 16 * act_slot<QT>(blk * 16 + lane / 2) + 8 * (lane & 1)) = o.codes;
  if constexpr (q8k) {
    if (lane == 0) ((float *)(dst + K))[blk] = o.d;
    if (lane % 2 == 0) ((int16_t *)(dst + K + act_d_bytes(true, K)))[blk * 16 + lane / 2] = (int16_t)o.sum16;
  } else {
    if (lane % 4 == 0) ((float *)(dst + K))[blk * 8 + lane / 4] = o.d;
  }
  return o;
}

// Weight rows r0 .. r1 of the slice w, every run's part of them rounded out to 16 bytes, asked for in the L2. (The last
// run's may reach up to 15 bytes past the slice: a matrix is followed by 16 bytes of its allocation.)
template <int QT>
__device__ __forceinline__ void prefetch_weight_rows(const uint8_t *w, uint64_t nblk, uint32_t K, uint32_t r0, uint32_t r1) {
  const uint32_t bpr = K / block_values(QT);
#pragma unroll
  for (uint32_t f = 0; f < nfields(QT); f++) {
    const uint32_t row = bpr * field(QT, f).size;
    const uint64_t run = run_offset(QT, f, nblk), at = (run + (uint64_t)r0 * row) & ~(uint64_t)15, end = (run + (uint64_t)r1 * row + 15) & ~(uint64_t)15;
    prefetch_l2_bulk(w + at, (uint32_t)(end - at));
  }
}

// The lists of a short step from its rows' experts (s_ids, kShortMax words, 0xFFFFFFFF past the last), by one CTA of 256
// threads: what k_router_topk_pack leaves for a step whose experts all stay below the tile kernels' threshold.
__device__ __forceinline__ void short_pack(const ShortRoute &rt, const uint32_t *s_ids) {
  __shared__ uint32_t s_groups[kShortMax];  // an expert's groups, at its first assignment
  const uint32_t A = rt.T * rt.K, tid = threadIdx.x;
  for (uint32_t e = tid; e < rt.NE; e += blockDim.x) {
    uint32_t n = 0, first = 0;
    for (uint32_t i = 0; i < A; i++) n += s_ids[i] == e, first += s_ids[i] < e;
    rt.o.cnt[e] = n, rt.o.base[e] = first;
  }
  uint32_t n = 0, first = 0, before = 0;
  const uint32_t e = tid < A ? s_ids[tid] : 0xFFFFFFFFu;
  const bool valid = e < rt.NE;
  if (tid < A) {
    for (uint32_t i = 0; i < A; i++) n += s_ids[i] == e, first += s_ids[i] < e, before += i < tid && s_ids[i] == e;
    s_groups[tid] = valid && before == 0 ? (n + rt.group_max - 1) / rt.group_max : 0;
    if (valid) rt.inv[tid] = first + before, rt.row_src[first + before] = tid / rt.K;
  }
  __syncthreads();
  if (valid && before == 0) {
    uint32_t tile = 0, group = 0;
    for (uint32_t i = 0; i < A; i++)
      if (s_ids[i] < e) tile += s_groups[i] != 0, group += s_groups[i];
    rt.o.tiles[tile] = MoeTile{e, e, first, n};
    for (uint32_t i = 0; i * rt.group_max < n; i++) rt.o.groups[group + i] = MoeGroup{e, first + i * rt.group_max, min(rt.group_max, n - i * rt.group_max)};
  }
  if (tid < 32) {
    uint32_t hit = 0, groups = 0, rows = 0;
    for (uint32_t i = tid; i < A; i += 32) hit += s_groups[i] != 0, groups += s_groups[i], rows += s_ids[i] < rt.NE;
    hit = __reduce_add_sync(0xffffffffu, hit), groups = __reduce_add_sync(0xffffffffu, groups), rows = __reduce_add_sync(0xffffffffu, rows);
    if (tid == 0) rt.o.counters[0] = hit, rt.o.counters[1] = groups, rt.o.counters[2] = hit, rt.o.counters[3] = rows, rt.o.counters[4] = 0, rt.o.counters[5] = 0, rt.o.counters[6] = 0;
  }
}

// The route of a short step by a CTA of 256 threads: its rows' experts into s_ids (kShortMax words); with `lists`, the
// step's ids, weights, gates and lists written too.
__device__ __forceinline__ void short_route(const ShortRoute &rt, uint32_t *s_ids, bool lists) {
  if (threadIdx.x < kShortMax) s_ids[threadIdx.x] = 0xFFFFFFFFu;  // a row whose logits are not numbers may have no K experts
  __syncthreads();
  const uint32_t warp = threadIdx.x / 32;
  if (warp < rt.T)
    router_topk_row(warp, rt.rl, RouterApprox{}, nullptr, rt.NE, rt.K, lists ? rt.ids : nullptr, lists ? rt.w : nullptr, rt.gs, nullptr,
                    (int32_t *)s_ids + warp * rt.K, nullptr);
  __syncthreads();
  if (lists) short_pack(rt, s_ids);
}

// The forms of k_expert_rows: the lists' groups; (gate/up, one or two rows) the top-k in the kernel; (down) rows
// quantised in the kernel.
enum RowsForm { ROWS_LISTED, ROWS_ROUTED, ROWS_QUANT };

// NMAT 2: h[row][r] = swiglu(gate_r . x, up_r . x); NMAT 1: y[row][r] = down_r . h. One CTA of 8 warps per (row tile,
// group); G lanes share a weight row (G = the row's units, up to 32), each taking UPL of its units (UPL 0: as many as
// the row has, found at run time). Launch: grid (R / (rows_per_cta * slabs), groups at most, CTAs that share a group), 256
// threads, dynamic shared memory M * act_row_stride and a codebook type's codebook.
//
// ROWS_ROUTED (NMAT 2, steps of one or two rows): no top-k or list kernel runs in front. Every CTA takes the top-k of the
// rows for itself, a warp a row (2 to 3 us, as long as it takes a kernel of its own, less that kernel's launch: 33.9 ->
// 29.2 us for one row of Q8_0); the grid's second extent is the assignments and one more. The CTAs of an expert's first
// assignment take all of its rows, those of its others leave; the last index's one CTA writes the lists. With more rows
// the CTAs that find their place and leave are too many (4 rows: 55 us against 29).
// ROWS_QUANT (NMAT 1, steps of a few rows): the rows come as f32 (act_f32) and every CTA quantises those it stages, so that no
// quantiser runs between the two products.
//
// Q6_K's forms for one and two rows are held to 128 registers, two CTAs an SM: left to itself the compiler takes up to 148 and
// one CTA is left (32 rows of Q6_K with Q8_0, 235 experts: 377 us against 308; one row of Q6_K 59 against 56). The other
// types' forms find their own balance (0: no minimum).
__host__ __device__ constexpr int rows_min_ctas(int qt, int m) { return qt == QT_Q6_K && m <= 2 ? 2 : 0; }
template <int QT, int NMAT, int M, int G, int UPL, int FORM>
__global__ void __launch_bounds__(256, rows_min_ctas(QT, M)) k_expert_rows(const ExpertRowsArgs a, const uint32_t *__restrict__ grid_global) {
  extern __shared__ __align__(16) uint8_t smem[];
  dependents_may_launch(), wait_for_predecessors();
  constexpr bool q8k = act_is_q8k(QT);
  uint32_t slot, start, n;
  constexpr bool QUANT = FORM == ROWS_QUANT, ROUTED = FORM == ROWS_ROUTED;
  [[maybe_unused]] __shared__ uint32_t s_ids[ROUTED ? kShortMax : 1], s_act[ROUTED ? M : 1];
  if constexpr (ROUTED) {
    const ShortRoute &rt = a.route;
    const uint32_t A = rt.T * rt.K, wp = threadIdx.x / 32, ln = threadIdx.x % 32;
    const bool lists = blockIdx.y == A;
    if (lists && blockIdx.x) return;
    short_route(rt, s_ids, lists);
    if (lists) return;
    // This assignment's expert, its rows and where its run starts, by every warp alike: at most 32 assignments, one a lane.
    const uint32_t e = s_ids[blockIdx.y], id = s_ids[ln], same = __ballot_sync(0xffffffffu, id == e);
    start = __popc(__ballot_sync(0xffffffffu, id < e));
    if (e >= rt.NE || blockIdx.y != (uint32_t)__ffs(same) - 1) return;
    slot = e, n = __popc(same);
    if (wp == 0 && id == e) s_act[__popc(same & ((1u << ln) - 1))] = ln / rt.K;
    __syncthreads();
  } else if (a.groups) {
    // Both loads go out together: the list is as long as the grid, so the entry can be read before the count says
    // whether it is one (a CTA's life is a chain of dependent loads; this takes one link out).
    const uint32_t ng = *a.ngroups;
    const MoeGroup g = a.groups[blockIdx.y];
    if (blockIdx.y >= ng) return;
    if (blockIdx.z * M >= g.n) return;
    slot = g.slot, start = g.start + blockIdx.z * M, n = min((uint32_t)M, g.n - blockIdx.z * M);
  } else {
    start = blockIdx.y * M;
    if (start >= a.dense_rows) return;
    slot = 0, n = min((uint32_t)M, a.dense_rows - start);
  }
  const uint32_t K = a.K, stride = act_row_stride(q8k, K), dsz = act_d_bytes(q8k, K);
  const uint32_t upr = K / Unit<QT>::kValues;  // units per weight row
  const uint64_t nblk = (uint64_t)a.R * (K / block_values(QT));
  const uint8_t *w0 = a.w0 + (uint64_t)slot * a.slice_bytes;
  const uint8_t *w1 = NMAT == 2 ? a.w1 + (uint64_t)slot * a.slice_bytes : nullptr;
  const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32, li = lane % G, sub = lane / G;
  constexpr uint32_t RPP = 32 / G;  // weight rows a warp takes per pass
  constexpr int NU = UPL > 0 ? UPL : 1;
  constexpr int RB = rows_batch(NMAT, NU, M, grid_words(QT) > 0);  // passes whose loads go out together
  using Raw = typename Unit<QT>::Raw;
  const uint32_t rows_per_warp = UPL > 0 ? RPP * RB : a.rows_per_cta / 8;
  // A CTA takes `slabs` slabs of 8 * rows_per_warp weight rows one after another, so that what it does once (being
  // launched, finding its group, staging the activations) is spread over more weight bytes.
  const uint32_t slabs = UPL > 0 && a.slabs > 1 ? a.slabs : 1, slab_rows = 8 * rows_per_warp;
  const uint32_t r_begin = blockIdx.x * slabs * slab_rows + warp * rows_per_warp;

  // With the row length known at compile time, every load of the warp's rows goes out first, before the activations
  // are staged: the weights come from HBM and their latency is the kernel's, so as many bytes as the registers hold
  // are put in flight at once.
  Raw raw[RB][NMAT][NU];
  auto fetch_slab = [&](uint32_t base) {
#pragma unroll
    for (int b = 0; b < RB; b++) {
      const uint32_t r = base + b * RPP + sub;
      if (r < a.R) {
#pragma unroll
        for (int j = 0; j < NU; j++) {
          raw[b][0][j] = Unit<QT>::fetch(w0, nblk, K, r, li + G * j, nullptr);
          if constexpr (NMAT == 2) raw[b][1][j] = Unit<QT>::fetch(w1, nblk, K, r, li + G * j, nullptr);
        }
      }
    }
  };
  if constexpr (UPL > 0) fetch_slab(r_begin);
  // What the CTA's warps will come to later is asked for in the L2 now, by one thread: a warp loads a slab, computes it and
  // only then loads the next, so without this HBM's latency stands in front of every slab.
  if (threadIdx.x == 0) {
    const uint32_t end = min(a.R, (blockIdx.x + 1) * slabs * slab_rows), from = min(end, blockIdx.x * slabs * slab_rows + (UPL > 0 ? slab_rows : 0));
    if (from < end) {
      prefetch_weight_rows<QT>(w0, nblk, K, from, end);
      if constexpr (NMAT == 2) prefetch_weight_rows<QT>(w1, nblk, K, from, end);
    }
  }

  uint32_t *grid = (uint32_t *)(smem + M * stride);
  if constexpr (grid_words(QT) > 0)
    for (uint32_t i = threadIdx.x; i < grid_words(QT); i += 256) grid[i] = grid_global[grid_offset(QT) + i];
  // The group's activation rows into shared memory; rows past n get zero scales, so they add nothing.
  if constexpr (QUANT)
    for (uint32_t i = warp; i < n * (K / 256); i += 8) {
      const uint32_t t = i / (K / 256), blk = i % (K / 256);
      const float4 *src = (const float4 *)(a.act_f32 + (uint64_t)(start + t) * K + blk * 256);
      const QuantLane o = stage_quantized<QT>(src[2 * lane], src[2 * lane + 1], blk, lane, smem + t * stride, K);
      if (blockIdx.x == 0 && a.codes.q) store_codes<q8k>(o, (uint64_t)(start + t) * (K / 256) + blk, lane, a.codes);
    }
  for (uint32_t t = 0; t < (uint32_t)M; t++) {
    uint8_t *dst = smem + t * stride;
    if (t < n) {
      if constexpr (QUANT) continue;
      uint64_t row;
      if constexpr (ROUTED)
        row = s_act[t];
      else
        row = a.act_row ? a.act_row[start + t] : start + t;
      const int4 *src = (const int4 *)(a.act.q + row * a.act.q_stride);
      const float *sd = (const float *)((const uint8_t *)a.act.d + row * a.act.d_stride);
      for (uint32_t i = threadIdx.x; i < K / 16; i += 256) ((int4 *)dst)[act_slot<QT>(i)] = src[i];
      if (q8k) {
        const int16_t *sb = (const int16_t *)((const uint8_t *)a.act.bs + row * a.act.bs_stride);
        for (uint32_t i = threadIdx.x; i < K / 256; i += 256) ((float *)(dst + K))[i] = sd[i];
        for (uint32_t i = threadIdx.x; i < K / 16; i += 256) ((int16_t *)(dst + K + dsz))[i] = sb[i];
      } else {
        for (uint32_t i = threadIdx.x; i < K / 32; i += 256) ((float *)(dst + K))[i] = sd[i];
      }
    } else {
      for (uint32_t i = threadIdx.x; i < dsz / 4; i += 256) ((float *)(dst + K))[i] = 0.0f;
    }
  }
  __syncthreads();

  auto finish = [&](float (&acc)[NMAT][M], uint32_t r) {
    // All M rows' sums, also where the group has fewer: leaving the loop at the group's last row made the whole kernel slower
    // (groups of up to eight, 1,000 rows without the tensor cores: Q8_0 4.79 ms with every row's, 5.15 without; Q4_K 8.41, 8.96).
#pragma unroll
    for (int t = 0; t < M; t++)
#pragma unroll
      for (int m = 0; m < NMAT; m++)
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) acc[m][t] += __shfl_xor_sync(0xffffffffu, acc[m][t], off);
    if (li == 0 && r < a.R) {
#pragma unroll
      for (int t = 0; t < M; t++)
        if ((uint32_t)t < n) {
          float v = acc[0][t];
          if constexpr (NMAT == 2) v = swiglu(acc[0][t], acc[1][t], a.limit);
          a.out[(uint64_t)(start + t) * a.out_stride + r] = v;
        }
    }
  };

  if constexpr (UPL > 0) {
    for (uint32_t sl = 0; sl < slabs; sl++) {
      const uint32_t base = r_begin + sl * slab_rows;
      if (sl > 0) fetch_slab(base);
#pragma unroll
      for (int b = 0; b < RB; b++) {
        const uint32_t r = base + b * RPP + sub;
        float acc[NMAT][M];
#pragma unroll
        for (int m = 0; m < NMAT; m++)
#pragma unroll
          for (int t = 0; t < M; t++) acc[m][t] = 0.0f;
        if (r < a.R) {
#pragma unroll
          for (int j = 0; j < NU; j++) {
            unit_dot<QT, M>(raw[b][0][j], K, li + G * j, smem, stride, acc[0], n, grid);
            if constexpr (NMAT == 2) unit_dot<QT, M>(raw[b][1][j], K, li + G * j, smem, stride, acc[1], n, grid);
          }
        }
        finish(acc, r);
      }
    }
  } else {
    for (uint32_t rr = 0; rr < rows_per_warp; rr += RPP) {
      const uint32_t r = r_begin + rr + sub;
      float acc[NMAT][M];
#pragma unroll
      for (int m = 0; m < NMAT; m++)
#pragma unroll
        for (int t = 0; t < M; t++) acc[m][t] = 0.0f;
      if (r < a.R) {
        for (uint32_t u = li; u < upr; u += G) {
          const Raw x0 = Unit<QT>::fetch(w0, nblk, K, r, u, nullptr);
          unit_dot<QT, M>(x0, K, u, smem, stride, acc[0], n, grid);
          if constexpr (NMAT == 2) {
            const Raw x1 = Unit<QT>::fetch(w1, nblk, K, r, u, nullptr);
            unit_dot<QT, M>(x1, K, u, smem, stride, acc[1], n, grid);
          }
        }
      }
      finish(acc, r);
    }
  }
}

// The down product of a step of one row with everything after it: out[t][r] = sum over k, in rank order, of w[t][k] *
// (down_r of the row's k-th expert . h), + gs[t] * s[t][r], + res[t][r]. In place of a quantiser, k_expert_rows and
// k_combine, whose launches such a step spends its time on: a warp takes an output row r for every assignment of the step,
// so a CTA holds all of the inner rows, which it quantises itself (the same 2 KB of f32 a row by every CTA, out of L2: what
// makes it the slower form already for two rows, whose experts it would also read once a row: the layer in Q8_0 62 us
// against 56, in Q2_0 80 against 64, of 2,560 x 768 values in Q4_K 92 against 78). The codes are left in q, d, bs too, in
// expert order, by the CTAs in turn. G lanes a weight row, UPL units of it a lane.
// Launch: grid by rows_per_warp * 8 output rows, 256 threads, dynamic shared memory A * act_row_stride + the codebook.
struct DownCombineArgs {
  const uint8_t *w;
  uint64_t slice_bytes;
  uint32_t K, R;               // values per weight row; weight rows
  uint32_t rows_per_warp;
  uint32_t T, used, NE;
  const float *h;              // [expert-order row][K]
  const int32_t *ids;
  const float *wk;
  const uint32_t *inv;
  const float *gs, *s, *res;   // s, res: null, not wanted
  float *out;                  // [T][R]
  QuantJob codes;
};
constexpr uint32_t kDownCombineMaxSmem = 100 * 1024;  // two CTAs an SM
__host__ __device__ constexpr uint32_t down_combine_smem(uint32_t qt, uint32_t rows, uint32_t K) {
  return rows * act_row_stride(act_is_q8k(qt), K) + 4 * grid_words(qt);
}
// Whether the kernel takes a step of `rows` assignments: its rows fit a CTA, and a weight row has at most 128 units.
__host__ __device__ constexpr bool down_combine_takes(uint32_t qt, uint32_t rows, uint32_t K) {
  const uint32_t unit = qt == QT_Q8_0 ? 16 : qt == QT_IQ3_S || qt == QT_IQ3_XXS || qt == QT_IQ2_S || qt == QT_Q2_0 ? 64 : 32;
  return K / unit <= 128 && down_combine_smem(qt, rows, K) <= kDownCombineMaxSmem;
}
template <int QT, int G, int UPL>
__global__ void __launch_bounds__(256) k_down_combine(const DownCombineArgs a, const uint32_t *__restrict__ grid_global) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ uint32_t s_ids[kShortMax], s_row[kShortMax];
  __shared__ float s_w[kShortMax], s_y[8][kShortMax];
  dependents_may_launch();
  constexpr bool q8k = act_is_q8k(QT);
  static_assert(down_combine_takes(QT, 1, 128 * Unit<QT>::kValues) == (down_combine_smem(QT, 1, 128 * Unit<QT>::kValues) <= kDownCombineMaxSmem) &&
                    !down_combine_takes(QT, 0, 129 * Unit<QT>::kValues),
                "the type's unit, as the host's rule has it");
  constexpr uint32_t RPP = 32 / G;
  constexpr int RB = rows_batch(1, UPL, 1, grid_words(QT) > 0);
  using Raw = typename Unit<QT>::Raw;
  const uint32_t A = a.T * a.used, K = a.K, stride = act_row_stride(q8k, K), upr = K / Unit<QT>::kValues;
  const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32, li = lane % G, sub = lane / G;
  const uint64_t nblk = (uint64_t)a.R * (K / block_values(QT));
  uint32_t *grid = (uint32_t *)(smem + A * stride);
  if constexpr (grid_words(QT) > 0)
    for (uint32_t i = threadIdx.x; i < grid_words(QT); i += 256) grid[i] = grid_global[grid_offset(QT) + i];
  wait_for_predecessors();
  if (threadIdx.x < A) {
    s_ids[threadIdx.x] = (uint32_t)a.ids[threadIdx.x], s_row[threadIdx.x] = a.inv[threadIdx.x], s_w[threadIdx.x] = a.wk[threadIdx.x];
    // An assignment without an expert (a row whose logits are not numbers) adds nothing.
    if (s_ids[threadIdx.x] >= a.NE || s_row[threadIdx.x] >= A) s_ids[threadIdx.x] = 0xFFFFFFFFu;
  }
  __syncthreads();
  Raw raw[RB][UPL];
  auto fetch = [&](uint32_t r, uint32_t a0) {
#pragma unroll
    for (int b = 0; b < RB; b++) {
      const uint32_t i = a0 + b * RPP + sub;
      if (r < a.R && i < A && s_ids[i] != 0xFFFFFFFFu) {
        const uint8_t *w = a.w + (uint64_t)s_ids[i] * a.slice_bytes;
#pragma unroll
        for (int j = 0; j < UPL; j++)
          if (li + G * j < upr) raw[b][j] = Unit<QT>::fetch(w, nblk, K, r, li + G * j, nullptr);
      }
    }
  };
  // The first weights are on their way while the inner rows are quantised.
  const uint32_t r0 = (blockIdx.x * 8 + warp) * a.rows_per_warp;
  fetch(r0, 0);
  for (uint32_t i = warp; i < A * (K / 256); i += 8) {
    const uint32_t p = i / (K / 256), blk = i % (K / 256);
    const float4 *src = (const float4 *)(a.h + (uint64_t)p * K + blk * 256);
    const QuantLane o = stage_quantized<QT>(src[2 * lane], src[2 * lane + 1], blk, lane, smem + p * stride, K);
    if (p % gridDim.x == blockIdx.x) store_codes<q8k>(o, (uint64_t)p * (K / 256) + blk, lane, a.codes);
  }
  __syncthreads();
  for (uint32_t rr = 0; rr < a.rows_per_warp && r0 + rr < a.R; rr++) {
    const uint32_t r = r0 + rr;
    for (uint32_t a0 = 0; a0 < A; a0 += RPP * RB) {
      if (rr | a0) fetch(r, a0);
#pragma unroll
      for (int b = 0; b < RB; b++) {
        const uint32_t i = a0 + b * RPP + sub;
        float acc = 0.0f;
        if (i < A && s_ids[i] != 0xFFFFFFFFu) {
#pragma unroll
          for (int j = 0; j < UPL; j++)
            if (li + G * j < upr) unit_dot<QT, 1>(raw[b][j], K, li + G * j, smem + s_row[i] * stride, stride, &acc, 1, grid);
        }
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
        if (li == 0 && i < A) s_y[warp][i] = acc;
      }
    }
    __syncwarp();
    if (lane < a.T) {
      float acc = 0.0f;
      for (uint32_t k = 0; k < a.used; k++) acc = fmaf(s_w[lane * a.used + k], s_y[warp][lane * a.used + k], acc);
      const uint64_t at = (uint64_t)lane * a.R + r;
      if (a.s) acc = fmaf(a.gs[lane], a.s[at], acc);
      if (a.res) acc += a.res[at];
      a.out[at] = acc;
    }
    __syncwarp();
  }
}

}  // namespace moe

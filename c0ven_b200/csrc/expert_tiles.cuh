// The experts' products for many rows per expert: a grouped GEMM on the 5th-generation tensor cores. A work item is 256
// weight rows of one expert and up to 256 of the rows routed to it; persistent pairs of CTAs, one CTA an SM, take items in turn.
// Decode warps turn the quantised blocks into f16 straight into shared memory in the tensor core's K-major
// core-matrix layout; one thread brings the rows' activations beside them with bulk-tensor (TMA) copies, 64 rows a
// copy, in the 128-byte-swizzled K-major layout; one lane of a warp issues tcgen05.mma with the weights as the M side and the rows as the N side (so a
// short tile costs a short instruction), accumulating f32 in tensor memory; epilogue warps read the accumulators back with
// tcgen05.ld, apply SwiGLU and store. This replaces the reference's moe_gate_up_t / moe_down_t
// (kernels/quant/qgemm.cl:88-239), whose tiles are 64 rows on Xe2's DPAS.
//
// Operands are IEEE f16, not bf16: the rows are the activations as the CPU path quantises them (q8_0 or q8_K,
// core/cpu/experts.cpp:166-168,229-237), dequantised; with f16's 11-bit significand the products stay within a few
// 1e-3 of that path's integer arithmetic, which bf16's 8 bits do not.
//
// Every wait on an mbarrier is bounded: a wait that runs out raises the CTA's abort flag and a global error word, the
// other waits return at once, and the CTA still frees its tensor memory before it exits.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "expert_rows.cuh"
#include "formats.h"

namespace moe {

constexpr uint32_t kTileM = 128;   // weight rows a CTA takes
constexpr uint32_t kTileN = 256;   // activation rows at most
constexpr uint32_t kTileK = 64;    // values of the contraction a stage holds
constexpr uint32_t kTileDecoders = 512;  // threads that decode weights: 16 warps, enough of them to hide their loads' latency
// Threads that turn accumulators into results: a warp per quarter of the weight rows, two for the down product, whose items are
// a quarter as long as gate's and up's for twice the results. That pays where tiles are full (the layer with one and with two:
// 32,768 rows of Q4_K 4,143 and 4,058 us; 8,192, skewed, 1,206 and 1,225, within what its runs differ by; 4,352 of IQ4_XS, 85 rows
// an expert, 892 and 897).
__host__ __device__ constexpr uint32_t tile_epilogue(int nmat) { return nmat == 1 ? 256 : 128; }
__host__ __device__ constexpr uint32_t tile_threads(int nmat) { return kTileDecoders + tile_epilogue(nmat) + 96; }  // and the rows' copy warp, the MMA warp, the quants' copy warp
constexpr uint32_t kTileBoxRows = 64;    // rows one bulk-tensor copy brings (the tensor map's box: 64 values x 64 rows)

struct ExpertTilesArgs {
  const uint8_t *w0, *w1;   // slot 0's slice of (gate, up) or (down, unused), runs layout
  uint64_t slice_bytes;
  uint32_t K, R;            // values per weight row; weight rows
                            // the activation rows, f16 [rows][K] in the order of the tiles, come through the tensor map
  const BigTile *tiles;     // null: dense_rows rows of slot 0 in tiles of kTileN
  const uint32_t *ntiles;
  uint32_t dense_rows;
  const uint32_t *gather_rows;  // not null: row r of the tiles' order is row gather_rows[r] of the map's tensor, whose box is
                                // one row (the copies gather four rows each); null: the same row, boxes of 64 rows
  void *out;                // out[expert-order row][r]: f32, or f16 when out_f16 is set
  uint32_t out_stride;
  uint32_t out_f16;
  float limit;
  uint32_t *error;          // set non-zero when a wait ran out
  // For types whose quants come by copy (quants_by_copy): maps over the quants runs of w0 and w1, (bytes of a row, rows,
  // expert slots), their box (a quant slot's bytes a row, 128 rows, 1 slot) (tensor_map.h: make_quants_map).
  CUtensorMap qmap[2];
};

namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// One bounded hardware wait: the warp sleeps until the phase completes or the hint (in ns) runs out.
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity, uint32_t hint_ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok != 0;
}
// Waits for the barrier's phase `parity` to complete, for about a second at most. False when it gave up or another
// thread of the CTA already had. The wait suspends the warp rather than spinning, so it takes no issue slots from the
// warps that decode.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t *abort, uint32_t *error) {
  if (mbar_test(bar, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
    if (mbar_try(bar, parity, 20000)) return true;
    if (*abort) return false;
    if (clock64() - t0 > 2000000000ll) {
      *abort = 1;
      atomicExch(error, 1u);
      return false;
    }
  }
}
// mbar_wait by a whole warp: every lane leaves it together, with the same answer.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile uint32_t *abort, uint32_t *error) {
  if (__all_sync(0xffffffffu, mbar_test(bar, parity))) return true;
  const long long t0 = clock64();
  for (;;) {
    if (__all_sync(0xffffffffu, mbar_try(bar, parity, 20000))) return true;
    const bool late = clock64() - t0 > 2000000000ll;
    if (__any_sync(0xffffffffu, late || *abort)) {
      if (late && !*abort) *abort = 1, atomicExch(error, 1u);
      return false;
    }
  }
}
// One lane of the warp, the same one every time.
__device__ __forceinline__ uint32_t elect_leader() {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r));
  return r;
}
// One arrival that also tells the barrier to expect `bytes` of bulk copies before its phase completes.
__device__ __forceinline__ void mbar_arrive_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Box (x .. x + 63 values, y .. y + 63 rows) of the map's tensor into shared memory at dst (1024-byte aligned); the
// bytes are counted on the barrier as they land. x * 2 bytes is a multiple of 16, as every bulk-tensor copy needs.
__device__ __forceinline__ void tma_load_rows(uint32_t dst_smem, const CUtensorMap *map, uint32_t x, uint32_t y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst_smem), "l"((uint64_t)map), "r"(x), "r"(y), "r"(bar)
               : "memory");
}
// Four rows y0 .. y3 of the map's tensor (its box one row of 64 values), values x .. x + 63 of each, into four
// consecutive 128-byte rows of shared memory at dst (512-byte aligned inside a 1024-byte aligned tile), swizzled as the
// tile's other rows are. The rows need not be neighbours: this is how a tile's rows are gathered by index. By a CTA of a pair,
// the bytes counted on a barrier that may be the other CTA's.
__device__ __forceinline__ void tma_gather4_rows_pair(uint32_t dst_smem, const CUtensorMap *map, uint32_t x, uint32_t y0, uint32_t y1,
                                                      uint32_t y2, uint32_t y3, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
      ::"r"(dst_smem), "l"((uint64_t)map), "r"(x), "r"(y0), "r"(y1), "r"(y2), "r"(y3), "r"(bar)
      : "memory");
}
// Box (x .. of the row's bytes, rows y .., expert slot z) of a weight matrix's quants run into shared memory at dst.
// x is a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_quants(uint32_t dst_smem, const CUtensorMap *map, uint32_t x, uint32_t y, uint32_t z, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
               ::"r"(dst_smem), "l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(bar)
               : "memory");
}
// --- A pair of CTAs (a cluster of two on the two SMs of a TPC) that share one product: tcgen05's cta_group::2. ---
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The shared::cluster address of the same place in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Arrivals on a barrier that may be the other CTA's (a shared::cluster address). What the arriving thread wrote for the
// tensor core to read has passed its own fence.proxy.async before; a release for the whole cluster on every arrival
// was measured to cost the decode warps a third of their rate and is left out, as in CUTLASS's pipelines for a pair.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_cluster(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cluster.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// All threads of both CTAs.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// tma_load_rows by a CTA of a pair: the bytes land in this CTA's shared memory and are counted on the barrier `bar`,
// which may be the other CTA's (a shared::cluster address).
__device__ __forceinline__ void tma_load_rows_pair(uint32_t dst_smem, const CUtensorMap *map, uint32_t x, uint32_t y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst_smem), "l"((uint64_t)map), "r"(x), "r"(y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// MMAs and commits are issued by one lane, `leader`, in code that the whole warp runs together: the instruction takes its
// descriptors from uniform registers, which the compiler can keep them in only where no lane goes its own way. (Issued in a branch
// for lane 0 an MMA of 96 rows took 173 clocks of that thread and one of 256 rows 200, by its own clock counts, for 48 and 128 of
// the tensor core's, and it waited for a tenth of them; so 152 and 182.)
// The pair's commit: one arrival on the barrier at this place in each CTA of the mask.
__device__ __forceinline__ void mma_commit_pair(uint32_t leader, uint32_t bar, uint32_t cta_mask) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %2, 0;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
      ::"r"(bar), "h"((uint16_t)cta_mask), "r"(leader)
      : "memory");
}
// D[tmem of both CTAs] (+)= A[256 rows: 128 in each CTA's shared memory] * B[n rows: half in each CTA's]^T, issued by
// one thread of the pair's first CTA; the descriptors name the same places in both.
__device__ __forceinline__ void mma_f16_pair(uint32_t leader, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %6, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u), "r"(leader)
      : "memory");
}

__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t leader, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      ::"r"(bar), "r"(leader)
      : "memory");
}
// D[tmem] (+)= A[smem] * B[smem]^T, f16 operands, f32 accumulate, M 128, K 16.
__device__ __forceinline__ void mma_f16(uint32_t leader, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(leader)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t *v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// The wait, naming the registers the loads fill: nothing that reads them can be scheduled before it.
__device__ __forceinline__ void tmem_ld_wait8(uint32_t *v) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7])
               :
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait16(uint32_t *v) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]),
                 "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])
               :
               : "memory");
}

// A K-major operand tile without swizzle: core matrices of 8 rows x 16 bytes, contiguous (128 bytes); the next 8
// values of the contraction 128 bytes on (the leading offset), the next 8 rows 1024 bytes on (the stride offset).
// Element (row, k) of a stage, k < 64: (row / 8) * 1024 + (k / 8) * 128 + (row % 8) * 16 + (k % 8) * 2.
constexpr uint32_t kLbo = 128, kSbo = 1024;
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(kLbo >> 4) << 16) | ((uint64_t)(kSbo >> 4) << 32) | (1ull << 46);
}
// The rows' tile as the bulk-tensor copies lay it: a row is 128 contiguous bytes (64 values) whose 16-byte pieces are
// swizzled by the row's low three bits; 8 rows 1024 bytes on. The next 16 values of the contraction: 32 bytes on.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// kind::f16 instruction descriptor: f32 accumulator, f16 A and B, both K-major, M 128, N n.
__device__ __forceinline__ uint32_t instr_desc(uint32_t n, uint32_t m = kTileM) { return (1u << 4) | ((n >> 3) << 17) | ((m >> 4) << 24); }

__device__ __forceinline__ void store_chunk(uint8_t *tile, uint32_t row, uint32_t kc, uint4 v) {
  *(uint4 *)(tile + (row >> 3) * kSbo + kc * kLbo + (row & 7) * 16) = v;
}

// Two bytes of x as f16 values 1024 + byte: the exponent byte 0x64 beside each.
__device__ __forceinline__ uint32_t bias_h2(uint32_t x, uint32_t sel) { return __byte_perm(x, 0x64646464u, sel); }
__device__ __forceinline__ __half2 as_h2(uint32_t u) { return *reinterpret_cast<__half2 *>(&u); }
__device__ __forceinline__ uint32_t as_u32(__half2 h) { return *reinterpret_cast<uint32_t *>(&h); }

__device__ __forceinline__ uint4 ldg16(const void *p) {
  uint4 v;
  asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}


__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Small integers as f16 without an int-to-float conversion: 0x6400 | v is 1024 + v for v < 1024.
__device__ __forceinline__ __half2 small_h2(uint32_t v) { return __hsub2(as_h2(0x64006400u | v | (v << 16)), as_h2(0x64006400u)); }

// ---------------------------------------------------------------------------------------------------------------
// Decoders. A stage is 64 values of every one of the tile's 128 weight rows, and a thread turns a whole row of it into f16,
// as two halves of 32 values: chunks 4 h .. 4 h + 3 of row m of the operand tile. All arithmetic is in f16 pairs;
// integers reach f16 through the exponent trick above, never through a conversion instruction.
//
// A type whose quants come by the threads' own loads is fetched in units of kUnitStages stages of a row, into registers,
// a unit ahead of the decode. A load whose lanes each read a row of their own costs the load pipe a wavefront a lane,
// whatever its width, so a unit is as much of a row as one round of wide loads brings: half a block of 256 values (two
// stages), whose codes, signs, high bits and scales are then 3 to 8 loads. (Fetched a stage at a time, in halves of 32,
// the same 128 values were 8 to 28 loads: 28 for Q6_K, 20 for IQ2_S and IQ3_S.) The unit of Q8_0 is one stage: two units of
// two in flight spill registers there, which cost more than the loads. Gate and up of IQ3_S and Q6_K spill too, 188 and 788 bytes of loads
// a thread, and gain all the same: the layer's time at 4,352 rows is 0.90 and 0.63 of what it was with halves.
template <int QT>
struct Decoder;

// Q8_0: w = d * q. A half is one block.
template <>
struct Decoder<QT_Q8_0> {
  static constexpr uint32_t kUnitStages = 1;
  static constexpr uint32_t kUnitBytes = 64;  // of the main quants run
  __device__ static __forceinline__ const uint8_t *quants_at(const uint8_t *s, uint32_t K, uint32_t r, uint32_t u) { return s + (uint64_t)r * K + 64 * u; }
  struct Raw {
    uint4 q[4];
    __half2 d;
  };
  __device__ static __forceinline__ Raw fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t u) {
    Raw x;
    const uint8_t *q = quants_at(s, K, r, u);
#pragma unroll
    for (int i = 0; i < 4; i++) x.q[i] = ldg16(q + 16 * i);
    x.d = __ldg((const __half2 *)((const __half *)(s + 32 * nblk) + (uint64_t)r * (K / 32) + 2 * u));
    return x;
  }
  template <int S>
  __device__ static __forceinline__ void store(const Raw &x, uint8_t *tile, uint32_t m, const uint32_t *) {
    const __half2 off = as_h2(0x64806480u);  // 1152 = 1024 + 128
#pragma unroll
    for (int c = 0; c < 8; c++) {  // a chunk of eight values
      const __half2 d2 = c < 4 ? __low2half2(x.d) : __high2half2(x.d);
      const uint4 &q = x.q[c / 2];
      const uint32_t u0 = (c & 1 ? q.z : q.x) ^ 0x80808080u, u1 = (c & 1 ? q.w : q.y) ^ 0x80808080u;  // int8 + 128
      uint4 o;
      o.x = as_u32(__hmul2(__hsub2(as_h2(bias_h2(u0, 0x4140)), off), d2)), o.y = as_u32(__hmul2(__hsub2(as_h2(bias_h2(u0, 0x4342)), off), d2));
      o.z = as_u32(__hmul2(__hsub2(as_h2(bias_h2(u1, 0x4140)), off), d2)), o.w = as_u32(__hmul2(__hsub2(as_h2(bias_h2(u1, 0x4342)), off), d2));
      store_chunk(tile, m, c, o);
    }
  }
};

// Q4_K: w = d * sc * q - dmin * m. A stage is 32 bytes of qs: their low nibbles are its first 32 values (sub-block 2c),
// their high nibbles its second 32 (sub-block 2c + 1). The two threads of a row's stage take 16 of the 32 bytes each,
// both nibbles: values 16 h .. 16 h + 15 of each sub-block, chunks 2 h, 2 h + 1 and 4 + 2 h, 5 + 2 h of the stage. The
// block's d, dmin and scales are one 16-byte piece, loaded once for its four stages.
template <>
struct Decoder<QT_Q4_K> {
  static constexpr uint32_t kUnitStages = 1;
  struct Hdr {
    uint4 v;  // d, dmin; then the 12 bytes of packed scales and minimums
  };
  struct Raw {
    uint4 q;
  };
  __device__ static __forceinline__ Hdr fetch_hdr(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t k0) {
    return Hdr{__ldg((const uint4 *)(s + 128 * nblk + 16 * ((uint64_t)r * (K / 256) + k0 / 256)))};
  }
  // The 6-bit scale and minimum of sub-blocks 2 c and 2 c + 1 (QUANT_FORMATS.md:386-392), each pair as two bytes of a word.
  __device__ static __forceinline__ void scales_of(const Hdr &x, uint32_t c, uint32_t &sc, uint32_t &mn) {
    // Bytes 2 c, 2 c + 1 of the three words of packed scales: words y (bytes 0-3), z (4-7), w (8-11).
    const uint32_t lo = c & 1 ? 0x7732u : 0x7710u;  // byte_perm selector for bytes 2 (c & 1), 2 (c & 1) + 1, zero-extended
    if (c < 2) {
      sc = __byte_perm(x.v.y, 0, lo) & 0x3F3Fu, mn = __byte_perm(x.v.z, 0, lo) & 0x3F3Fu;
    } else {
      const uint32_t p = __byte_perm(x.v.w, 0, lo), a = __byte_perm(x.v.y, 0, lo), b = __byte_perm(x.v.z, 0, lo);
      sc = (p & 0x0F0Fu) | ((a >> 2) & 0x3030u), mn = ((p >> 4) & 0x0F0Fu) | ((b >> 2) & 0x3030u);
    }
  }
  // The stage's 32 bytes of a row, both nibbles. A byte beside the exponent byte 0x64 is the f16 value 1024 + byte: 1024 + q
  // for a low nibble, 1024 + 16 q for a high nibble left in place. q comes out exactly (v - 1024, or v / 16 - 64 in one
  // fused step); then w = a * q + c with a = d * sc and c = -dmin * m, each a product of two f16 numbers rounded once,
  // taken for both sub-blocks by one instruction and once for the stage.
  __device__ static __forceinline__ void store(const Hdr &hd, const Raw (&x)[2], uint8_t *tile, uint32_t m, uint32_t k0) {
    uint32_t sc, mn;
    scales_of(hd, (k0 % 256) / 64, sc, mn);
    const __half2 dm = as_h2(hd.v.x), k1024 = as_h2(0x64006400u), k16th = as_h2(0x2C002C00u), km64 = as_h2(0xD400D400u);  // 1024, 1/16, -64
    const __half2 A = __hmul2(__low2half2(dm), __hsub2(as_h2(bias_h2(sc, 0x4140)), k1024));
    const __half2 C = __hmul2(__high2half2(dm), __hsub2(k1024, as_h2(bias_h2(mn, 0x4140))));
    const __half2 A0 = __low2half2(A), A1 = __high2half2(A), C0 = __low2half2(C), C1 = __high2half2(C);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t w[4] = {x[h].q.x, x[h].q.y, x[h].q.z, x[h].q.w};
      uint32_t lo[8], hi[8];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint32_t l = w[i] & 0x0F0F0F0Fu, g = w[i] & 0xF0F0F0F0u;
        lo[2 * i] = as_u32(__hfma2(__hsub2(as_h2(bias_h2(l, 0x4140)), k1024), A0, C0));
        lo[2 * i + 1] = as_u32(__hfma2(__hsub2(as_h2(bias_h2(l, 0x4342)), k1024), A0, C0));
        hi[2 * i] = as_u32(__hfma2(__hfma2(as_h2(bias_h2(g, 0x4140)), k16th, km64), A1, C1));
        hi[2 * i + 1] = as_u32(__hfma2(__hfma2(as_h2(bias_h2(g, 0x4342)), k16th, km64), A1, C1));
      }
      store_chunk(tile, m, 2 * h, make_uint4(lo[0], lo[1], lo[2], lo[3]));
      store_chunk(tile, m, 2 * h + 1, make_uint4(lo[4], lo[5], lo[6], lo[7]));
      store_chunk(tile, m, 4 + 2 * h, make_uint4(hi[0], hi[1], hi[2], hi[3]));
      store_chunk(tile, m, 5 + 2 * h, make_uint4(hi[4], hi[5], hi[6], hi[7]));
    }
  }
};

// Q6_K: w = d * scales[v / 16] * (q - 32). A unit is half a block: 64 bytes of ql, whose low nibbles are the first stage's
// values and whose high ones the second's, 32 bytes of qh (bits 0, 1 and 2, 3 of them the first stage's halves, 4, 5 and
// 6, 7 the second's) and eight scales, two a half.
template <>
struct Decoder<QT_Q6_K> {
  static constexpr uint32_t kUnitStages = 2;
  static constexpr uint32_t kUnitBytes = 64;  // of the main quants run
  __device__ static __forceinline__ const uint8_t *quants_at(const uint8_t *s, uint32_t K, uint32_t r, uint32_t u) { return s + (uint64_t)r * (K / 2) + 64 * u; }
  struct Raw {
    uint4 l[4], h[2];
    uint2 sc;
    __half d;
  };
  __device__ static __forceinline__ Raw fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t u) {
    const uint64_t blk = (uint64_t)r * (K / 256) + u / 2;
    const uint32_t hh = u % 2;
    Raw x;
    const uint8_t *ql = quants_at(s, K, r, u), *qh = s + 128 * nblk + 64 * blk + 32 * hh;
#pragma unroll
    for (int i = 0; i < 4; i++) x.l[i] = ldg16(ql + 16 * i);
    x.h[0] = ldg16(qh), x.h[1] = ldg16(qh + 16);
    x.sc = __ldg((const uint2 *)(s + 192 * nblk + 16 * blk + 8 * hh));
    x.d = __ldg((const __half *)(s + 208 * nblk) + blk);
    return x;
  }
  template <int S>
  __device__ static __forceinline__ void store(const Raw &x, uint8_t *tile, uint32_t m, const uint32_t *) {
    const __half2 d2 = __half2half2(x.d), off = as_h2(0x64206420u), o128 = as_h2(0x64806480u);  // 1056 = 1024 + 32; 1152
    const uint32_t b[8] = {x.h[0].x, x.h[0].y, x.h[0].z, x.h[0].w, x.h[1].x, x.h[1].y, x.h[1].z, x.h[1].w};
    const uint32_t scu = (S ? x.sc.y : x.sc.x) ^ 0x80808080u;  // int8 + 128
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t l[8] = {x.l[2 * h].x, x.l[2 * h].y, x.l[2 * h].z, x.l[2 * h].w, x.l[2 * h + 1].x, x.l[2 * h + 1].y, x.l[2 * h + 1].z, x.l[2 * h + 1].w};
      const __half2 ds0 = __hmul2(d2, __hsub2(as_h2(bias_h2(scu, h ? 0x4242 : 0x4040)), o128));
      const __half2 ds1 = __hmul2(d2, __hsub2(as_h2(bias_h2(scu, h ? 0x4343 : 0x4141)), o128));
#pragma unroll
      for (int c = 0; c < 4; c++) {
        uint4 o;
        uint32_t *p = &o.x;
#pragma unroll
        for (int k = 0; k < 2; k++) {
          const int i = 2 * c + k;
          const uint32_t q = ((l[i] >> (4 * S)) & 0x0F0F0F0Fu) | (((b[i] >> (4 * S + 2 * h)) & 0x03030303u) << 4);
          const __half2 ds = i < 4 ? ds0 : ds1;
          p[2 * k] = as_u32(__hmul2(__hsub2(as_h2(bias_h2(q, 0x4140)), off), ds));
          p[2 * k + 1] = as_u32(__hmul2(__hsub2(as_h2(bias_h2(q, 0x4342)), off), ds));
        }
        store_chunk(tile, m, 4 * h + c, o);
      }
    }
  }
};

// IQ3_S: w = d * (1 + 2 s) * grid[index][i] * sign. A half is one sub-block of 32: 8 bytes of qs, a byte of qh, 4 of
// signs, a nibble of scale; a unit is four of them. The codebook is in shared memory.
template <>
struct Decoder<QT_IQ3_S> {
  static constexpr uint32_t kUnitStages = 2;
  static constexpr uint32_t kUnitBytes = 32;  // of the main quants run
  __device__ static __forceinline__ const uint8_t *quants_at(const uint8_t *s, uint32_t K, uint32_t r, uint32_t u) { return s + (uint64_t)r * (K / 4) + 32 * u; }
  struct Raw {
    uint4 qs[2], sg;
    uint32_t qh;
    uint16_t sc;
    __half d;
  };
  __device__ static __forceinline__ Raw fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t u) {
    const uint64_t blk = (uint64_t)r * (K / 256) + u / 2;
    const uint32_t hh = u % 2;
    Raw x;
    const uint8_t *qs = quants_at(s, K, r, u);
    x.qs[0] = ldg16(qs), x.qs[1] = ldg16(qs + 16);
    x.sg = ldg16(s + 64 * nblk + 32 * blk + 16 * hh);
    x.qh = __ldg((const uint32_t *)(s + 96 * nblk + 8 * blk + 4 * hh));
    x.sc = __ldg((const uint16_t *)(s + 104 * nblk + 4 * blk + 2 * hh));
    x.d = __ldg((const __half *)(s + 108 * nblk) + blk);
    return x;
  }
  template <int S>
  __device__ static __forceinline__ void store(const Raw &x, uint8_t *tile, uint32_t m, const uint32_t *grid) {
    const __half2 d2 = __half2half2(x.d), off = as_h2(0x64006400u);
    const uint32_t qs[4] = {x.qs[S].x, x.qs[S].y, x.qs[S].z, x.qs[S].w};
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const __half2 ls = small_h2(2 * (((uint32_t)x.sc >> (8 * S + 4 * h)) & 0xF) + 1);
      const uint32_t qh = x.qh >> (16 * S + 8 * h), sg = S ? (h ? x.sg.w : x.sg.z) : (h ? x.sg.y : x.sg.x);
#pragma unroll
      for (int c = 0; c < 4; c++) {
        uint4 o;
        uint32_t *p = &o.x;
#pragma unroll
        for (int j = 0; j < 2; j++) {
          const int k = 2 * c + j;
          const uint32_t g = grid[((qs[2 * h + k / 4] >> (8 * (k & 3))) & 0xFF) | (((qh >> k) & 1u) << 8)];
          const uint32_t nib = (sg >> (4 * k)) & 0xF;
          // The sign bit of each f16: values 4k, 4k + 1 from the nibble's bits 0, 1; 4k + 2, 4k + 3 from bits 2, 3.
          const uint32_t s01 = ((nib & 1u) << 15) | ((nib & 2u) << 30), s23 = ((nib & 4u) << 13) | ((nib & 8u) << 28);
          p[2 * j] = as_u32(__hmul2(__hmul2(__hsub2(as_h2(bias_h2(g, 0x4140)), off), ls), d2)) ^ s01;
          p[2 * j + 1] = as_u32(__hmul2(__hmul2(__hsub2(as_h2(bias_h2(g, 0x4342)), off), ls), d2)) ^ s23;
        }
        store_chunk(tile, m, 4 * h + c, o);
      }
    }
  }
};

// Four codebook bytes (a word of values below 128) times sc as f16 with the nibble's signs, into o[0], o[1].
__device__ __forceinline__ void grid_word_to_f16(uint32_t g, uint32_t nib, __half2 sc, uint32_t *o) {
  const __half2 off = as_h2(0x64006400u);
  // The sign bit of each f16: values 0, 1 from the nibble's bits 0, 1; 2, 3 from bits 2, 3.
  const uint32_t s01 = ((nib & 1u) << 15) | ((nib & 2u) << 30), s23 = ((nib & 4u) << 13) | ((nib & 8u) << 28);
  o[0] = as_u32(__hmul2(__hsub2(as_h2(bias_h2(g, 0x4140)), off), sc)) ^ s01;
  o[1] = as_u32(__hmul2(__hsub2(as_h2(bias_h2(g, 0x4342)), off), sc)) ^ s23;
}

// IQ3_XXS: w = d * (0.5 + s) / 2 * grid[index][i] * sign. A half is one sub-block of 32: 8 bytes of indices and its
// word of four 7-bit sign indices and the scale; a unit is four of them. The codebook is in shared memory.
template <>
struct Decoder<QT_IQ3_XXS> {
  static constexpr uint32_t kUnitStages = 2;
  static constexpr uint32_t kUnitBytes = 32;  // of the main quants run
  __device__ static __forceinline__ const uint8_t *quants_at(const uint8_t *s, uint32_t K, uint32_t r, uint32_t u) { return s + (uint64_t)r * (K / 4) + 32 * u; }
  struct Raw {
    uint4 qs[2], w32;
    __half d;
  };
  __device__ static __forceinline__ Raw fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t u) {
    const uint64_t blk = (uint64_t)r * (K / 256) + u / 2;
    const uint32_t hh = u % 2;
    Raw x;
    const uint8_t *qs = quants_at(s, K, r, u);
    x.qs[0] = ldg16(qs), x.qs[1] = ldg16(qs + 16);
    x.w32 = ldg16(s + 64 * nblk + 32 * blk + 16 * hh);
    x.d = __ldg((const __half *)(s + 96 * nblk) + blk);
    return x;
  }
  template <int S>
  __device__ static __forceinline__ void store(const Raw &x, uint8_t *tile, uint32_t m, const uint32_t *grid) {
    const uint32_t qs[4] = {x.qs[S].x, x.qs[S].y, x.qs[S].z, x.qs[S].w};
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t w32 = S ? (h ? x.w32.w : x.w32.z) : (h ? x.w32.y : x.w32.x);
      // d * (2 s + 1) / 4, rounded to f16 once.
      const __half2 sc = __float2half2_rn(__half2float(x.d) * (float)(2 * (w32 >> 28) + 1) * 0.25f);
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const uint32_t k7 = (w32 >> (7 * c)) & 127u, sbyte = k7 | ((__popc(k7) & 1u) << 7);
        const uint32_t word = qs[2 * h + c / 2] >> (16 * (c & 1));
        uint32_t o[4];
        grid_word_to_f16(grid[word & 0xFF], sbyte & 0xF, sc, o), grid_word_to_f16(grid[(word >> 8) & 0xFF], sbyte >> 4, sc, o + 2);
        store_chunk(tile, m, 4 * h + c, make_uint4(o[0], o[1], o[2], o[3]));
      }
    }
  }
};

// IQ2_S: w = d * (0.5 + s) / 4 * grid[index][i] * sign. A half is one sub-block of 32: four groups of 8 values, each a
// 10-bit index (a byte of qs, two bits of the sub-block's qh byte) and a byte of signs; a scale nibble per two groups.
// A unit is four sub-blocks.
template <>
struct Decoder<QT_IQ2_S> {
  static constexpr uint32_t kUnitStages = 2;
  static constexpr uint32_t kUnitBytes = 16;  // of the main quants run
  __device__ static __forceinline__ const uint8_t *quants_at(const uint8_t *s, uint32_t K, uint32_t r, uint32_t u) { return s + (uint64_t)r * (K / 8) + 16 * u; }
  struct Raw {
    uint4 qs, sg;
    uint32_t qh, sc;
    __half d;
  };
  __device__ static __forceinline__ Raw fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t u) {
    const uint64_t blk = (uint64_t)r * (K / 256) + u / 2;
    const uint32_t hh = u % 2;
    Raw x;
    x.qs = ldg16(quants_at(s, K, r, u));
    x.sg = ldg16(s + 32 * nblk + 32 * blk + 16 * hh);
    x.qh = __ldg((const uint32_t *)(s + 64 * nblk + 8 * blk + 4 * hh));
    x.sc = __ldg((const uint32_t *)(s + 72 * nblk + 8 * blk + 4 * hh));
    x.d = __ldg((const __half *)(s + 80 * nblk) + blk);
    return x;
  }
  template <int S>
  __device__ static __forceinline__ void store(const Raw &x, uint8_t *tile, uint32_t m, const uint32_t *grid) {
    const float d8 = __half2float(x.d) * 0.125f;  // d * (2 s + 1) / 8
    const uint2 *grid2 = (const uint2 *)grid;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t sc = x.sc >> (16 * S + 8 * h), qh = x.qh >> (16 * S + 8 * h);
      const uint32_t qs = S ? (h ? x.qs.w : x.qs.z) : (h ? x.qs.y : x.qs.x), sg = S ? (h ? x.sg.w : x.sg.z) : (h ? x.sg.y : x.sg.x);
      const __half2 sc_lo = __float2half2_rn(d8 * (float)(2 * (sc & 0xF) + 1)), sc_hi = __float2half2_rn(d8 * (float)(2 * ((sc >> 4) & 0xF) + 1));
#pragma unroll
      for (int g = 0; g < 4; g++) {
        const uint2 e = grid2[((qs >> (8 * g)) & 0xFF) | (((qh >> (2 * g)) & 3u) << 8)];
        const uint32_t sb = (sg >> (8 * g)) & 0xFF;
        uint32_t o[4];
        grid_word_to_f16(e.x, sb & 0xF, g < 2 ? sc_lo : sc_hi, o), grid_word_to_f16(e.y, sb >> 4, g < 2 ? sc_lo : sc_hi, o + 2);
        store_chunk(tile, m, 4 * h + g, make_uint4(o[0], o[1], o[2], o[3]));
      }
    }
  }
};

// Sixteen table values (four words of signed bytes) times d2 as f16, into o[0 .. 7].
__device__ __forceinline__ void int8x16_to_f16(const uint32_t (&w)[4], __half2 d2, uint32_t *o) {
  const __half2 off = as_h2(0x64806480u);  // 1152 = 1024 + 128
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const uint32_t u = w[j] ^ 0x80808080u;  // int8 + 128
    o[2 * j] = as_u32(__hmul2(__hsub2(as_h2(bias_h2(u, 0x4140)), off), d2));
    o[2 * j + 1] = as_u32(__hmul2(__hsub2(as_h2(bias_h2(u, 0x4342)), off), d2));
  }
}
// A block or sub-block of 32 four-bit codes (16 bytes: values 0 .. 15 in the low nibbles, 16 .. 31 in the high ones)
// through the table, times d2, into chunks 4 h .. 4 h + 3 of the row. The permutes that put the exponent byte beside two of the
// looked-up bytes take every other one, so they part low nibbles from high ones too.
__device__ __forceinline__ void iq4_store32(const uint4 &q, __half2 d2, uint8_t *tile, uint32_t m, uint32_t h) {
  const __half2 off = as_h2(0x64806480u);  // 1152 = 1024 + 128
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
  uint32_t lo[8], hi[8];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint2 v = iq4_pairs<128>(w[i]);
    lo[2 * i] = as_u32(__hmul2(__hsub2(as_h2(bias_h2(v.x, 0x4240)), off), d2)), lo[2 * i + 1] = as_u32(__hmul2(__hsub2(as_h2(bias_h2(v.y, 0x4240)), off), d2));
    hi[2 * i] = as_u32(__hmul2(__hsub2(as_h2(bias_h2(v.x, 0x4341)), off), d2)), hi[2 * i + 1] = as_u32(__hmul2(__hsub2(as_h2(bias_h2(v.y, 0x4341)), off), d2));
  }
#pragma unroll
  for (int c = 0; c < 2; c++) {
    store_chunk(tile, m, 4 * h + c, make_uint4(lo[4 * c], lo[4 * c + 1], lo[4 * c + 2], lo[4 * c + 3]));
    store_chunk(tile, m, 4 * h + 2 + c, make_uint4(hi[4 * c], hi[4 * c + 1], hi[4 * c + 2], hi[4 * c + 3]));
  }
}

// Q2_0: w = (q - 1) * d. A stage is one block of 64, 16 bytes.
template <>
struct Decoder<QT_Q2_0> {
  static constexpr uint32_t kUnitStages = 2;
  static constexpr uint32_t kUnitBytes = 32;  // of the main quants run
  __device__ static __forceinline__ const uint8_t *quants_at(const uint8_t *s, uint32_t K, uint32_t r, uint32_t u) { return s + (uint64_t)r * (K / 4) + 32 * u; }
  struct Raw {
    uint4 q[2];
    __half2 d;
  };
  __device__ static __forceinline__ Raw fetch(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t u) {
    Raw x;
    const uint8_t *q = quants_at(s, K, r, u);
    x.q[0] = ldg16(q), x.q[1] = ldg16(q + 16);
    x.d = __ldg((const __half2 *)((const __half *)(s + 16 * nblk) + (uint64_t)r * (K / 64) + 2 * u));
    return x;
  }
  template <int S>
  __device__ static __forceinline__ void store(const Raw &x, uint8_t *tile, uint32_t m, const uint32_t *) {
    const __half2 d2 = S ? __high2half2(x.d) : __low2half2(x.d);
    const uint32_t q[4] = {x.q[S].x, x.q[S].y, x.q[S].z, x.q[S].w};
#pragma unroll
    for (int i = 0; i < 4; i++) {  // 16 values a word
      uint32_t w[4], o[8];
#pragma unroll
      for (int j = 0; j < 4; j++) w[j] = q2_bytes((q[i] >> (8 * j)) & 0xFF);
      int8x16_to_f16(w, d2, o);
      store_chunk(tile, m, 2 * i, make_uint4(o[0], o[1], o[2], o[3])), store_chunk(tile, m, 2 * i + 1, make_uint4(o[4], o[5], o[6], o[7]));
    }
  }
};

// IQ4_NL: w = d * table[q], blocks of 32 with a scale each; a header is the eight scales of 256 values.
template <>
struct Decoder<QT_IQ4_NL> {
  static constexpr uint32_t kUnitStages = 1;
  struct Hdr {
    uint4 d;
  };
  struct Raw {
    uint4 q;
  };
  __device__ static __forceinline__ Hdr fetch_hdr(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t k0) {
    return Hdr{__ldg((const uint4 *)((const __half *)(s + 16 * nblk) + (uint64_t)r * (K / 32) + k0 / 32))};
  }
  __device__ static __forceinline__ void store(const Hdr &hd, const Raw (&x)[2], uint8_t *tile, uint32_t m, uint32_t k0) {
    const uint32_t c = k0 % 256 / 64;
    const __half2 d = as_h2(c & 2 ? (c & 1 ? hd.d.w : hd.d.z) : (c & 1 ? hd.d.y : hd.d.x));
    iq4_store32(x[0].q, __low2half2(d), tile, m, 0), iq4_store32(x[1].q, __high2half2(d), tile, m, 1);
  }
};

// IQ4_XS: w = d * (ls - 32) * table[q], sub-blocks of 32 with a 6-bit ls each.
template <>
struct Decoder<QT_IQ4_XS> {
  static constexpr uint32_t kUnitStages = 1;
  struct Hdr {
    uint32_t sl, sh;  // the eight sub-blocks' low nibbles; their high pairs of bits
    __half d;
  };
  struct Raw {
    uint4 q;
  };
  __device__ static __forceinline__ Hdr fetch_hdr(const uint8_t *s, uint64_t nblk, uint32_t K, uint32_t r, uint32_t k0) {
    const uint64_t blk = (uint64_t)r * (K / 256) + k0 / 256;
    return Hdr{__ldg((const uint32_t *)(s + 128 * nblk) + blk), __ldg((const uint16_t *)(s + 132 * nblk) + blk), __ldg((const __half *)(s + 134 * nblk) + blk)};
  }
  __device__ static __forceinline__ void store(const Hdr &hd, const Raw (&x)[2], uint8_t *tile, uint32_t m, uint32_t k0) {
    const uint32_t c = k0 % 256 / 64, sl = hd.sl >> (8 * c), sh = hd.sh >> (4 * c);
    // d * (ls - 32) rounded to f16 once; ls - 32 is in -32 .. 31, exact in f16.
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t ls = ((sl >> (4 * h)) & 0xF) | (((sh >> (2 * h)) & 3) << 4);
      iq4_store32(x[h].q, __float2half2_rn(__half2float(hd.d) * (float)((int)ls - 32)), tile, m, h);
    }
  }
};

}  // namespace tc


// Whether a type's quants reach the decode warps through a ring in shared memory filled by bulk-tensor copies, rather
// than by the warps' own global loads (whose one-row-per-lane pattern costs the load pipe 32 wavefronts an
// instruction). Q4_K, IQ4_XS and IQ4_NL: their quants are one run of K / 2 bytes a row, which a 3-D map (bytes of the
// row, rows, expert slots) covers. (IQ4_XS with IQ4_NL, 4,352 rows of the benchmark's layer, by the threads' own loads and
// the table's values parted by permutes of their own: gate and up 448 us, 417 so; the layer 985 and 944.)
__host__ __device__ constexpr bool quants_by_copy(uint32_t qt) { return qt == QT_Q4_K || qt == QT_IQ4_XS || qt == QT_IQ4_NL; }

// What a decode thread loads of a block beside the quants the ring brings.
template <int QT, bool = quants_by_copy(QT)>
struct HeaderOf {
  using type = typename tc::Decoder<QT>::Hdr;
};
template <int QT>
struct HeaderOf<QT, false> {
  struct type {};
};

// The values a stage holds. The stages of an item follow one another through the decode groups, stage it going to group
// it % groups; where a group's unit is two stages, they are the units of `groups` groups at a time, first stages first, so
// that a thread finds both stages of a unit in the registers it filled with one round of loads. A row whose units the
// groups do not divide ends with half a round: as many stages as there are groups, taken in the row's order, one each.
// No group so goes more than `groups` stages without one of its own: its wait on a stage's empty barrier tells the
// phases apart only if its last stage lies no further back than the ring is long.
template <int QT, uint32_t GROUPS>
struct StageMap {
  static constexpr uint32_t kUnit = tc::Decoder<QT>::kUnitStages, kRound = GROUPS * kUnit;
  __device__ static __forceinline__ uint32_t first_value(uint32_t it, uint32_t KT) {
    if constexpr (kUnit == 1) return it * kTileK;
    const uint32_t r0 = it / kRound * kRound, i = it - r0;
    return (KT - r0 >= kRound ? r0 + i % GROUPS * kUnit + i / GROUPS : it) * kTileK;
  }
};

// Shared memory of a CTA: the stages (NMAT weight tiles of 16 KB and half a row tile, 16 KB, each), then (for types whose
// quants come by copy) a ring of two quant slots, then the barriers, then a codebook type's codebook.
// A quant slot holds, for every weight row of the item, the quants of one stage per decode group: 32 bytes a stage in these
// types of four bits a value, so 64 bytes a row with two groups (64-byte swizzle) and 128 with four (128-byte swizzle).
template <int QT, int NMAT>
struct TileSmem {
  static constexpr uint32_t kStages = NMAT == 2 ? 4 : 6;
  static constexpr uint32_t kXRows = kTileN / 2;                                      // a CTA of a pair holds half the rows' tile
  static constexpr uint32_t kWBytes = kTileM * kTileK * 2, kXBytes = kXRows * kTileK * 2;
  static constexpr uint32_t kStageBytes = NMAT * kWBytes + kXBytes;
  static constexpr uint32_t kGroups = kTileDecoders / (NMAT * kTileM);                // decode groups: 2 or 4
  static constexpr uint32_t kQRowBytes = kGroups * 32;                                // a row's bytes in a quant slot
  static constexpr uint32_t kQMatBytes = kTileM * kQRowBytes, kQSlotBytes = NMAT * kQMatBytes, kQSlots = 2;
  static constexpr uint32_t kQuants = kStages * kStageBytes;
  static constexpr uint32_t kBarriers = kQuants + (quants_by_copy(QT) ? kQSlots * kQSlotBytes : 0);
  // full[kStages], empty[kStages], accumulators full[2], empty[2], empty after a two-buffer item, quant slots full[2],
  // empty[2]; tmem address; abort
  static constexpr uint32_t kGrid = kBarriers + 256;                                  // the codebook: 1, 2 or 8 KB
  static constexpr uint32_t kBytes = kGrid + 4 * grid_words(QT) + 1024;               // and room to align the base to 1024
  static_assert(kBytes <= 227 * 1024, "a CTA's shared memory");
};

// SwiGLU with the fast exponential and division: the tensor-core path's results already differ from the CPU path's
// in the last bits of f16 products, so full-precision expf buys nothing here.
__device__ __forceinline__ float swiglu_fast(float g, float u, float limit) {
  if (limit > 0.0f) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
  }
  return __fdividef(g, 1.0f + __expf(-g)) * u;
}


// The tile a work item belongs to.
struct ItemTile {
  uint32_t slot, start, count;
};
__device__ __forceinline__ ItemTile item_tile(const ExpertTilesArgs &a, uint32_t ti) {
  if (a.tiles) {
    const BigTile t = a.tiles[ti];
    return ItemTile{t.slot, t.start, t.count};
  }
  const uint32_t start = ti * kTileN;
  return ItemTile{0, start, min(kTileN, a.dense_rows - start)};
}

// NMAT 2: out = swiglu(gate x, up x); NMAT 1: out = down h. Persistent: the grid is one CTA per SM (fewer when there is
// less work), in clusters of two on the two SMs of a TPC. Such a pair is one unit of work: it takes the items dealt to it round by
// round; item i is pair of weight-row tiles i % RTU of big tile i / RTU, so neighbouring pairs share a tile's
// activations in L2. Five roles: 16 decode warps (quants to f16 weights in shared memory), 4 or 8 epilogue warps
// (accumulators to the result), a warp whose first lane issues the bulk-tensor copies of the rows' activations (the
// whole warp when the rows are gathered by index), the warp that owns tensor memory and runs the MMAs in step, one elected
// lane of it issuing them, and a warp whose first lane issues the copies of the quants for types that take them through the
// ring. A warp arrives on a barrier once, by one lane.
//
// Tensor memory is two buffers of 256 columns. An item of at most 128 rows (any item, for NMAT 1) takes one buffer,
// alternately, so the epilogue warps drain item i while the MMAs of item i + 1 run and the decode warps never stop. A
// gate/up item of more than 128 rows needs both buffers (gate in one, up in the other): the MMAs of the next item
// wait for its epilogue, and to keep that short the decode warps join the epilogue warps for it.
// Dynamic shared memory TileSmem::kBytes.
template <int QT, int NMAT>
__global__ void __launch_bounds__(tile_threads(NMAT), 1) k_expert_tiles(const __grid_constant__ ExpertTilesArgs a,
                                                                  const __grid_constant__ CUtensorMap act_map,
                                                                  const uint32_t *__restrict__ grid_global) {
  using namespace tc;
  using SM = TileSmem<QT, NMAT>;
  using Dec = Decoder<QT>;
  using Raw = typename Dec::Raw;
  constexpr uint32_t S = SM::kStages, kCols = 512;
  constexpr uint32_t kDW = kTileDecoders / 32, kEW = tile_epilogue(NMAT) / 32, kCopyWarp = kDW + kEW, kMmaWarp = kCopyWarp + 1, kQuantWarp = kMmaWarp + 1;
  // A decode thread takes a whole row of a stage, 64 values as two halves of 32, so that what a stage costs a thread
  // beside the arithmetic (the barrier round trip, the addresses, the block's scales) is paid once per 64 values. A
  // stage's NMAT * 128 rows are one group of threads; the 512 decode threads form 2 groups (two matrices) or 4 (one),
  // and group g takes stages g, g + groups, ...
  constexpr uint32_t kGroupThreads = NMAT * kTileM, kDecGroups = kTileDecoders / kGroupThreads;
  static_assert(kDecGroups <= S, "a decode group waits on the phase before the last of a stage it may not have seen (StageMap)");
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);

  const uint32_t K = a.K, KT = K / kTileK;
  const uint32_t ntiles = a.tiles ? *a.ntiles : (a.dense_rows + kTileN - 1) / kTileN;
  // A pair's item is 256 weight rows (128 decoded by each CTA) times the tile's rows, of which each CTA brings half into its own
  // shared memory; the first CTA's MMA warp issues one tcgen05.mma.cta_group::2 for both, which reads both halves and writes each
  // CTA's 128 weight rows of the product into that CTA's tensor memory. What a CTA's shared memory carries per flop
  // is a single CTA's weights but only half its rows, and shared-memory bandwidth is what bounded the kernel by single CTAs.
  const uint32_t rank = cluster_ctarank();
  const uint32_t unit = blockIdx.x / 2, nunits = gridDim.x / 2;
  const uint32_t RTU = a.R / (2 * kTileM);  // a big tile's items
  const uint32_t nitems = ntiles * RTU;
  const uint32_t magic = item_magic(RTU);  // a big tile's number without a division (the launch bounds the tiles)
  auto tile_of_item = [&](uint32_t item) { return RTU > 1 ? __umulhi(item, magic) : item; };
  if (unit >= nitems) return;  // both CTAs of a pair alike
  const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  uint64_t *bars = (uint64_t *)(smem + SM::kBarriers);
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](uint32_t s) { return bar0 + 8 * s; };
  auto empty_bar = [&](uint32_t s) { return bar0 + 8 * (S + s); };
  auto acc_full = [&](uint32_t b) { return bar0 + 8 * (2 * S + b); };
  auto acc_empty = [&](uint32_t b) { return bar0 + 8 * (2 * S + 2 + b); };
  const uint32_t acc_empty_wide = bar0 + 8 * (2 * S + 4);
  auto q_full = [&](uint32_t b) { return bar0 + 8 * (2 * S + 5 + b); };
  auto q_empty = [&](uint32_t b) { return bar0 + 8 * (2 * S + 7 + b); };
  uint32_t *tmem_slot = (uint32_t *)(bars + 2 * S + 9);
  volatile uint32_t *abort = tmem_slot + 1;
  uint32_t *grid = (uint32_t *)(smem + SM::kGrid);

  // A stage is full when every decode warp has stored its weights (one arrival a warp) and the rows' copies have landed
  // (the copy thread's arrival states their bytes; the copy unit counts them off). An accumulator buffer is empty again
  // when the epilogue warps have read it; after an item that took both buffers, also when the decode warps have.
  if (tid == 0) {
    // In a pair the first CTA's full, accumulator-empty barriers take both CTAs' arrivals.
    constexpr uint32_t kCtas = 2;
    for (uint32_t s = 0; s < S; s++) mbar_init(full_bar(s), kCtas * (kDW / kDecGroups + 1)), mbar_init(empty_bar(s), 1);
    for (uint32_t b = 0; b < 2; b++) mbar_init(acc_full(b), 1), mbar_init(acc_empty(b), kCtas * kEW);
    mbar_init(acc_empty_wide, kCtas * kDW);
    for (uint32_t b = 0; b < 2; b++) mbar_init(q_full(b), 1), mbar_init(q_empty(b), kDW);
    *abort = 0;
    fence_barrier_init();
  }
  if constexpr (grid_words(QT) > 0)
    for (uint32_t i = tid; i < grid_words(QT); i += blockDim.x) grid[i] = grid_global[grid_offset(QT) + i];
  if (warp == kMmaWarp) tmem_alloc_pair(smem_u32(tmem_slot), kCols);  // the same warp of both CTAs, the same place for the address
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // the other CTA's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  bool ok = true;
  // The first CTA's barriers, as the pair's other CTA names them (for the first CTA itself: its own).
  const uint32_t bar0_lead = map_to_cta(bar0, 0);
  auto full_lead = [&](uint32_t s) { return bar0_lead + 8 * s; };
  auto acc_empty_lead = [&](uint32_t b) { return bar0_lead + 8 * (2 * S + 2 + b); };
  const uint32_t acc_empty_wide_lead = bar0_lead + 8 * (2 * S + 4);
  // The weight rows of an item that this CTA decodes and drains.
  auto item_rows0 = [&](uint32_t item) { return ((item - tile_of_item(item) * RTU) * 2u + rank) * kTileM; };

  // CTA b's item of round r: the items come expert by expert for the experts with full tiles, then the short tiles of
  // the others by falling row count, and the rounds deal them boustrophedon (b, then G - 1 - b, ...), so that every CTA
  // gets a like share of long and short items. kNoItem past the end; a CTA's last round may have no item for it while others still have one.
  constexpr uint32_t kNoItem = 0xFFFFFFFFu;
  auto item_at = [&](uint32_t rnd) {
    const uint32_t base = rnd * nunits;
    const uint32_t i = base + ((rnd & 1) ? nunits - 1 - unit : unit);
    return i < nitems ? i : kNoItem;
  };

  // Every role walks the same items and keeps the same books: how often each buffer has been used (the parity of its
  // barriers' phases), which buffer the next one-buffer item takes, and how many two-buffer items there have been.
  uint32_t use0 = 0, use1 = 0, next_buf = 0, wides = 0;  // two scalars, not an array: they stay in registers
  auto use_of = [&](uint32_t b) { return b ? use1 : use0; };
  auto use_inc = [&](uint32_t b) { use0 += b == 0, use1 += b == 1; };
  auto is_wide = [&](uint32_t count) { return NMAT == 2 && count > kTileN / 2; };

  // Columns q (this warp's quarter of the weight rows: TMEM lanes 32 q ..) of chunks slot, slot + nslots, ... of W rows
  // each, from the accumulators at column colg (and colu, the up product) to the result. A lane holds one weight row's
  // values for the chunk's W rows; for each row the warp's lanes store 32 consecutive values: in f32 one a lane, in f16 the even
  // lanes one row's and the odd ones the next's, two a lane. The address of a chunk is worked out once and stepped by the row stride: what the loop costs
  // per value is a conversion and a store, in f16 half a shuffle and half a store.
  // The loads of a warp's next chunk are in flight while it converts and stores the one before (two sets of
  // registers): what a chunk costs is then its instructions, not tensor memory's latency, which alone had the down
  // product's epilogue warps, four of them then, take longer over an item than its MMAs do.
  auto drain = [&](const ItemTile &t, uint32_t r0, uint32_t colg, uint32_t colu, uint32_t slot, uint32_t nslots) {
    constexpr int W = NMAT == 2 ? 8 : 16;
    const uint32_t q = warp % 4, r = r0 + 32 * q + lane, nch = ((t.count + 15) & ~15u) / W;
    const uint32_t lanes = tmem_base + ((32 * q) << 16);
    auto load = [&](uint32_t c, uint32_t *g, uint32_t *u) {
      if constexpr (NMAT == 2)
        tmem_ld8(lanes + colg + W * c, g), tmem_ld8(lanes + colu + W * c, u);
      else
        tmem_ld16(lanes + colg + W * c, g);
    };
    auto wait = [&](uint32_t *g, uint32_t *u) {
      if constexpr (NMAT == 2)
        tmem_ld_wait8(g), tmem_ld_wait8(u);
      else
        tmem_ld_wait16(g);
    };
    auto store = [&](uint32_t c, const uint32_t *g, const uint32_t *u) {
      if (W * c >= t.count) return;           // a chunk of rows past the tile's (the rows are rounded up to 16)
      const uint32_t left = t.count - W * c;  // rows of the chunk that exist
      float v[W];
#pragma unroll
      for (int j = 0; j < W; j++) {
        v[j] = __uint_as_float(g[j]);
        if constexpr (NMAT == 2) v[j] = swiglu_fast(v[j], __uint_as_float(u[j]), a.limit);
      }
      const uint64_t at = (uint64_t)(t.start + W * c) * a.out_stride + r;
      if (a.out_f16) {
        // Two lanes that hold neighbouring weight rows share out two result rows: the even one stores both values of the first,
        // the odd one of the second, four bytes each.
        const uint32_t odd = lane & 1, sel = odd ? 0x3276u : 0x5410u;
        uint32_t *p = (uint32_t *)((__half *)a.out + at + (uint64_t)odd * a.out_stride - odd);
#pragma unroll
        for (int j = 0; j < W; j += 2, p += a.out_stride) {
          const uint32_t mine = as_u32(__floats2half2_rn(v[j], v[j + 1])), theirs = __shfl_xor_sync(0xffffffffu, mine, 1);
          if (left >= (uint32_t)W || j + odd < left) *p = __byte_perm(mine, theirs, sel);
        }
      } else {
        float *p = (float *)a.out + at;
        if (left >= (uint32_t)W) {
#pragma unroll
          for (int j = 0; j < W; j++) p[(uint64_t)j * a.out_stride] = v[j];
        } else {
#pragma unroll
          for (int j = 0; j < W; j++)
            if ((uint32_t)j < left) p[(uint64_t)j * a.out_stride] = v[j];
        }
      }
    };
    uint32_t gA[W], gB[W], uA[NMAT == 2 ? W : 1], uB[NMAT == 2 ? W : 1];
    uint32_t c = slot;
    if (c >= nch) return;
    load(c, gA, uA);
    for (;;) {
      wait(gA, uA);
      uint32_t cn = c + nslots;
      if (cn < nch) load(cn, gB, uB);
      store(c, gA, uA);
      if (cn >= nch) break;
      c = cn, cn = c + nslots;
      wait(gB, uB);
      if (cn < nch) load(cn, gA, uA);
      store(c, gB, uB);
      if (cn >= nch) break;
      c = cn;
    }
  };

  if (warp < kDW) {
    // Decode warps. 8 consecutive threads take the 8 rows of a core matrix, so a quarter-warp's 16-byte stores fill 128
    // contiguous bytes.
    const uint64_t nblk = (uint64_t)a.R * (K / block_values(QT));
    const uint32_t first = tid / kGroupThreads, mat = (tid % kGroupThreads) / kTileM, m = tid % kTileM;
    uint32_t li = 0;
    // For types whose quants come by copy, the one thing a decode thread still loads itself is a block's header, and it
    // asks for it a block ahead (across items too), so that no stage begins by waiting for it: hdr_ahead holds the
    // header of the next block the thread will decode.
    [[maybe_unused]] typename HeaderOf<QT>::type hdr_ahead;
    if constexpr (quants_by_copy(QT)) {
      const uint32_t i0 = item_at(0);
      if (i0 != kNoItem && first < KT) {
        const ItemTile t0 = item_tile(a, tile_of_item(i0));
        hdr_ahead = Dec::fetch_hdr((mat == 0 ? a.w0 : a.w1) + (uint64_t)t0.slot * a.slice_bytes, nblk, K, item_rows0(i0) + m,
                                   (first * kTileK) & ~255u);
      }
    }
    for (uint32_t rnd = 0, item; (item = item_at(rnd)) != kNoItem && ok; rnd++, li++) {
      const ItemTile t = item_tile(a, tile_of_item(item));
      const uint32_t r0 = item_rows0(item);
      const uint8_t *wm = (mat == 0 ? a.w0 : a.w1) + (uint64_t)t.slot * a.slice_bytes;
      // The next item's weights and rows, known early: its first header is asked for at this item's last stage.
      const uint32_t item_after = quants_by_copy(QT) ? item_at(rnd + 1) : kNoItem;
      ItemTile t_after{0, 0, 0};
      if (item_after != kNoItem) t_after = item_tile(a, tile_of_item(item_after));
      auto stage_begin = [&](uint32_t it, uint32_t &s) {
        const uint32_t g = li * KT + it, use_s = g / S;
        s = g % S;
        if (use_s > 0) ok = mbar_wait(empty_bar(s), (use_s - 1) & 1, abort, a.error);
        if (ok) tc_fence_after();
        return ok;
      };
      auto stage_end = [&](uint32_t s) {
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(full_lead(s));
      };
      auto tile_of = [&](uint32_t s) { return smem + s * SM::kStageBytes + mat * SM::kWBytes; };
      if constexpr (quants_by_copy(QT)) {
        // This thread's stages: first, first + kDecGroups, ...; the quants wait in shared memory, so nothing is loaded ahead but
        // a block's scales, kept for the thread's later stages there.
        uint32_t blk_fetched = 0xFFFFFFFFu;
        typename Dec::Hdr hdr;
        for (uint32_t it = first; it < KT && ok; it += kDecGroups) {
          const uint32_t k0 = it * kTileK;
          // The header asked for a block ago is this block's; the one after it is asked for now.
          if (it == first || k0 / 256 != blk_fetched) hdr = hdr_ahead, blk_fetched = k0 / 256;
          const uint32_t it2 = it + kDecGroups;
          if (it2 < KT) {
            if (it2 * kTileK / 256 != blk_fetched) hdr_ahead = Dec::fetch_hdr(wm, nblk, K, r0 + m, (it2 * kTileK) & ~255u);
          } else if (item_after != kNoItem) {
            hdr_ahead = Dec::fetch_hdr((mat == 0 ? a.w0 : a.w1) + (uint64_t)t_after.slot * a.slice_bytes, nblk, K,
                                       item_rows0(item_after) + m, (first * kTileK) & ~255u);
          }
          // The stage's 32 bytes of this row from the quant ring: slot qn holds one stage per group, this group's at
          // bytes 32 * first of the row, its 16-byte pieces swizzled by the row as the copy laid them.
          const uint32_t qn = li * (KT / kDecGroups) + it / kDecGroups, qb = qn % SM::kQSlots;
          ok = mbar_wait(q_full(qb), (qn / SM::kQSlots) & 1, abort, a.error);
          if (!ok) break;
          const uint8_t *row = smem + SM::kQuants + qb * SM::kQSlotBytes + mat * SM::kQMatBytes + m * SM::kQRowBytes;
          const uint32_t sw = SM::kQRowBytes == 64 ? (m >> 1) & 3 : m & 7;
          Raw raw[2];
          raw[0].q = *(const uint4 *)(row + 16 * ((2 * first) ^ sw));
          raw[1].q = *(const uint4 *)(row + 16 * ((2 * first + 1) ^ sw));
          // These reads are the generic proxy's and the copy that refills the slot is the async proxy's: without the
          // fence the copy was seen to overtake them (a few 128-byte lines of a slot read as the next stage's quants,
          // run to run different). The fence orders the reads before whatever the arrival below lets loose.
          fence_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(q_empty(qb));
          uint32_t s;
          if (!stage_begin(it, s)) break;
          Dec::store(hdr, raw, tile_of(s), m, k0);
          stage_end(s);
        }
      } else {
        // This thread's units: first, first + kDecGroups, ...; one is loaded while the one before it decodes. In a round cut
        // short (half of one: StageMap) the thread takes one stage of the unit its stage falls into.
        constexpr uint32_t U = Dec::kUnitStages;
        const uint32_t units = KT / U, whole = units / kDecGroups * kDecGroups, last = whole + first / U;
        Raw raw[2];
        auto one_stage = [&](auto half, const Raw &x, uint32_t it) {
          uint32_t s;
          if (!stage_begin(it, s)) return;
          Dec::template store<decltype(half)::value>(x, tile_of(s), m, grid);
          stage_end(s);
        };
        auto fetch = [&](Raw &x, uint32_t u) {
          const uint32_t v = u < whole ? u : last;
          if (v >= units) return;
          x = Dec::fetch(wm, nblk, K, r0 + m, v);
          // The main run's lines come from HBM the first time an expert is touched: one request a 128-byte line for the L2,
          // a whole number of lines and at least three units of every group's ahead.
          constexpr uint32_t kLine = 128 / Dec::kUnitBytes, kAhead = (3 * kDecGroups + kLine - 1) / kLine * kLine;
          if (v % kLine == 0 && v + kAhead < units) prefetch_l2(Dec::quants_at(wm, K, r0 + m, v + kAhead));
        };
        auto unit_step = [&](const Raw &x, uint32_t u) {
          if (u < whole) {
            one_stage(std::integral_constant<int, 0>{}, x, (u - first) * U + first);
            if constexpr (U == 2)
              if (ok) one_stage(std::integral_constant<int, 1>{}, x, (u - first) * U + kDecGroups + first);
          } else if constexpr (U == 2) {
            const uint32_t it = whole * U + first;
            if (it >= KT) return;
            if (first % 2)
              one_stage(std::integral_constant<int, 1>{}, x, it);
            else
              one_stage(std::integral_constant<int, 0>{}, x, it);
          }
        };
        // The first lines of a row's quants are asked for an item ahead, so that an item does not begin by waiting for HBM.
        const uint32_t item_next = item_at(rnd + 1);
        if (first == 0 && item_next != kNoItem) {
          const ItemTile tn = item_tile(a, tile_of_item(item_next));
          const uint8_t *wn = (mat == 0 ? a.w0 : a.w1) + (uint64_t)tn.slot * a.slice_bytes;
          for (uint32_t u = 0; u < units && u < 3 * kDecGroups; u += 128 / Dec::kUnitBytes) prefetch_l2(Dec::quants_at(wn, K, item_rows0(item_next) + m, u));
        }
        const uint32_t rounds = (units + kDecGroups - 1) / kDecGroups;
        fetch(raw[0], first);
        for (uint32_t j = 0; j < rounds && ok; j += 2) {
          if (j + 1 < rounds) fetch(raw[1], first + (j + 1) * kDecGroups);
          unit_step(raw[0], first + j * kDecGroups);
          if (!ok || j + 1 >= rounds) break;
          if (j + 2 < rounds) fetch(raw[0], first + (j + 2) * kDecGroups);
          unit_step(raw[1], first + (j + 1) * kDecGroups);
        }
      }
      if (is_wide(t.count)) {
        // Both buffers: the next item's MMAs wait for this epilogue, so these warps take four fifths of it.
        if (ok) ok = mbar_wait(acc_full(0), use0 & 1, abort, a.error);
        if (ok) ok = mbar_wait(acc_full(1), use1 & 1, abort, a.error);
        if (ok) {
          tc_fence_after();
          drain(t, r0, 0, kTileN, warp / 4, kDW / 4 + 1);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(acc_empty_wide_lead);
        }
        use0++, use1++, wides++;
      } else {
        use_inc(next_buf), next_buf ^= 1;
      }
    }
  } else if (warp < kDW + kEW) {
    // Epilogue warps: warp w reads TMEM lanes 32 (w % 4) .., its quarter of the weight rows.
    uint32_t li = 0;
    for (uint32_t rnd = 0, item; (item = item_at(rnd)) != kNoItem && ok; rnd++, li++) {
      const ItemTile t = item_tile(a, tile_of_item(item));
      const uint32_t r0 = item_rows0(item);
      if (is_wide(t.count)) {
        if (ok) ok = mbar_wait(acc_full(0), use0 & 1, abort, a.error);
        if (ok) ok = mbar_wait(acc_full(1), use1 & 1, abort, a.error);
        if (!ok) break;
        tc_fence_after();
        drain(t, r0, 0, kTileN, kDW / 4, kDW / 4 + 1);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(acc_empty_lead(0)), mbar_arrive_cluster(acc_empty_lead(1));
        use0++, use1++, wides++;
      } else {
        const uint32_t b = next_buf;
        ok = mbar_wait(acc_full(b), use_of(b) & 1, abort, a.error);
        if (!ok) break;
        tc_fence_after();
        drain(t, r0, b * kTileN, b * kTileN + kTileN / 2, (warp - kDW) / 4, kEW / 4);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(acc_empty_lead(b));
        use_inc(b), next_buf ^= 1;
      }
    }
  } else if (warp == kCopyWarp) {
    if (a.gather_rows) {
      // The copy warp, gathering: the tile's rows are scattered over the activations (row r of the expert order is row
      // gather_rows[r] of the map's tensor) and a copy brings four of them: up to 32 copies a stage, one a lane. A lane keeps its
      // row indices for the whole item. Rows past the tile's count repeat its last row; their columns of the result are dropped.
      uint32_t li = 0;
      for (uint32_t rnd = 0, item; (item = item_at(rnd)) != kNoItem && ok; rnd++, li++) {
        const ItemTile t = item_tile(a, tile_of_item(item));
        const uint32_t half = ((t.count + 15) & ~15u) / 2, ncopies = (half + 3) / 4;
        uint32_t idx[4];
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) idx[j] = a.gather_rows[t.start + min(rank * half + 4 * lane + j, t.count - 1)];
        for (uint32_t it = 0; it < KT && ok; it++) {
          const uint32_t g = li * KT + it, s = g % S, use_s = g / S;
          if (lane == 0) {
            if (use_s > 0) ok = mbar_wait(empty_bar(s), (use_s - 1) & 1, abort, a.error);
            if (ok) mbar_arrive_expect_cluster(full_lead(s), ncopies * 4 * kTileK * 2);
          }
          ok = __shfl_sync(0xffffffffu, ok, 0);
          if (!ok) break;
          const uint32_t xt = smem_u32(smem + s * SM::kStageBytes) + NMAT * SM::kWBytes, x0 = StageMap<QT, kDecGroups>::first_value(it, KT);
          if (lane < ncopies) tma_gather4_rows_pair(xt + lane * 4 * kTileK * 2, &act_map, x0, idx[0], idx[1], idx[2], idx[3], full_lead(s));
        }
      }
      if (!ok && lane == 0) {
        const long long t0 = clock64();
        while (clock64() - t0 < 400000) {
        }
      }
      __syncwarp();
    } else if (lane == 0) {
      // The copy thread: per stage, the 64 values of the tile's rows, 64 rows a copy, in the swizzled layout. A copy may
      // run past the tile's rows into the next expert's, or past the tensor (zeros): those columns of the result are dropped.
      uint32_t li = 0;
      for (uint32_t rnd = 0, item; (item = item_at(rnd)) != kNoItem && ok; rnd++, li++) {
        const ItemTile t = item_tile(a, tile_of_item(item));
        // A CTA of a pair brings its half of the rows the instruction takes (the rows rounded up to 16): the first
        // CTA the first half.
        const uint32_t half = ((t.count + 15) & ~15u) / 2;
        const uint32_t row0 = t.start + rank * half, nbox = (half + kTileBoxRows - 1) / kTileBoxRows;
        for (uint32_t it = 0; it < KT && ok; it++) {
          const uint32_t g = li * KT + it, s = g % S, use_s = g / S;
          if (use_s > 0) ok = mbar_wait(empty_bar(s), (use_s - 1) & 1, abort, a.error);
          if (!ok) break;
          const uint32_t xt = smem_u32(smem + s * SM::kStageBytes) + NMAT * SM::kWBytes, x0 = StageMap<QT, kDecGroups>::first_value(it, KT);
          mbar_arrive_expect_cluster(full_lead(s), nbox * kTileBoxRows * kTileK * 2);
          for (uint32_t i = 0; i < nbox; i++)
            tma_load_rows_pair(xt + i * kTileBoxRows * kTileK * 2, &act_map, x0, row0 + i * kTileBoxRows, full_lead(s));
        }
      }
      if (!ok) {
        // Copies already issued may still be on their way: give them time to land before the CTA leaves.
        const long long t0 = clock64();
        while (clock64() - t0 < 400000) {
        }
      }
    }
  } else if (warp == kQuantWarp) {
    if (quants_by_copy(QT) && lane == 0) {
    // The quants' copy thread (a warp of its own: sharing a warp with the MMAs' issue cost the tile kernels 8 %): a quant slot, one stage per decode group for every weight row of the item, as soon
    // as the decode warps have read the slot's last contents; it runs ahead of the stages by the ring's two slots.
    uint32_t li = 0;
    for (uint32_t rnd = 0, item; (item = item_at(rnd)) != kNoItem && ok; rnd++, li++) {
      const ItemTile t = item_tile(a, tile_of_item(item));
      for (uint32_t j = 0; j < KT / kDecGroups && ok; j++) {
        const uint32_t qn = li * (KT / kDecGroups) + j, qb = qn % SM::kQSlots, use_q = qn / SM::kQSlots;
        if (use_q > 0) ok = mbar_wait(q_empty(qb), (use_q - 1) & 1, abort, a.error);
        if (!ok) break;
        const uint32_t dst = smem_u32(smem + SM::kQuants + qb * SM::kQSlotBytes);
        mbar_arrive_expect(q_full(qb), SM::kQSlotBytes);
        for (uint32_t mt = 0; mt < (uint32_t)NMAT; mt++)
          tma_load_quants(dst + mt * SM::kQMatBytes, &a.qmap[mt], j * SM::kQRowBytes, item_rows0(item), t.slot, q_full(qb));
      }
    }
    if (!ok) {
      const long long t0 = clock64();
      while (clock64() - t0 < 400000) {
      }
    }
    }
  } else if (rank == 0) {
    // The MMA warp (of a pair's first CTA), one lane of which issues: per stage, four K steps of 16 for each matrix; the
    // commit frees the stage when they are done, in both CTAs of a pair.
    const uint32_t leader = elect_leader();
    auto wait_lead = [&](uint32_t bar, uint32_t parity) { return mbar_wait_warp(bar, parity, abort, a.error); };
    auto mma = [&](uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) { mma_f16_pair(leader, d, da, db, idesc, acc); };
    auto commit = [&](uint32_t bar) { mma_commit_pair(leader, bar, 3); };
    const uint32_t stages = smem_u32(smem);
    uint32_t s = 0, phase = 0;
    bool after_wide = false;
    for (uint32_t rnd = 0, item; (item = item_at(rnd)) != kNoItem && ok; rnd++) {
      const ItemTile t = item_tile(a, tile_of_item(item));
      const uint32_t idesc = instr_desc((t.count + 15) & ~15u, 2 * kTileM);
      const bool wide = is_wide(t.count);
      const uint32_t b = next_buf, colg = tmem_base + (wide ? 0 : b * kTileN), colu = colg + (wide ? kTileN : kTileN / 2);
      // The buffers this item writes must have been read: by the epilogue warps, and after a two-buffer item by the
      // decode warps too.
      if (after_wide) ok = wait_lead(acc_empty_wide, (wides - 1) & 1);
      after_wide = false;
      for (uint32_t bb = 0; bb < 2 && ok; bb++)
        if ((wide || bb == b) && use_of(bb) > 0) ok = wait_lead(acc_empty(bb), (use_of(bb) - 1) & 1);
      for (uint32_t it = 0; it < KT && ok; it++) {
        ok = wait_lead(full_bar(s), phase);
        if (!ok) break;
        tc_fence_after();
        const uint32_t stage = stages + s * SM::kStageBytes, xt = stage + NMAT * SM::kWBytes;
#pragma unroll
        for (uint32_t k = 0; k < kTileK / 16; k++) {
          const uint64_t db = smem_desc_sw128(xt + 32 * k);
          mma(colg, smem_desc(stage + 2 * k * kLbo), db, idesc, (it | k) != 0);
          if constexpr (NMAT == 2) mma(colu, smem_desc(stage + SM::kWBytes + 2 * k * kLbo), db, idesc, (it | k) != 0);
        }
        commit(empty_bar(s));
        if (++s == S) s = 0, phase ^= 1;
      }
      if (!ok) break;
      if (wide) {
        commit(acc_full(0)), commit(acc_full(1));
        use0++, use1++, wides++, after_wide = true;
      } else {
        commit(acc_full(b));
        use_inc(b), next_buf ^= 1;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  // Neither CTA of a pair may leave (or free tensor memory) while the other may still read its shared memory or write
  // its tensor memory.
  cluster_sync();
  if (warp == kMmaWarp) {
    __syncwarp();
    tc_fence_after();
    tmem_free_pair(tmem_base, kCols);
  }
}

// act_map: the activation rows, f16 [rows][a.K] in the order of the tiles (tensor_map.h).
struct LaunchCtx;
template <int QT, int NMAT>
cudaError_t launch_expert_tiles(const ExpertTilesArgs &a, const CUtensorMap &act_map, uint32_t max_tiles, const uint32_t *grid_global,
                                const LaunchCtx &ctx, cudaStream_t st);

}  // namespace moe

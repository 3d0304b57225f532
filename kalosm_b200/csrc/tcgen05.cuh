// PTX wrappers of the 5th-generation tensor cores (tcgen05.mma, tensor memory loads and stores, commit), bounded
// mbarrier waits and tensor-map copies, shared by the prompt-pass kernels.
#pragma once

#include <cuda.h>

#include "qgemv_common.cuh"

namespace {

// Waits for a phase of an mbarrier, with a limit; false: it or another role of the CTA gave up.
__device__ __forceinline__ bool x_wait(uint32_t bar, uint32_t parity, volatile int* dead, int* status) {
  for (int it = 0; it < (1 << 22); ++it) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return true;
    if ((it & 255) == 255 && *dead) return false;
  }
  *dead = 1;
  if (status) atomicExch(status, FB200_ERR_TIMEOUT);
  return false;
}
// The same for a whole warp, which leaves it together: the vote keeps what follows uniform. (Lanes left to themselves drift apart,
// and one that is held up in a later wait can find the phase of the earlier one overtaken.)
__device__ __forceinline__ bool w_wait(uint32_t bar, uint32_t parity, volatile int* dead, int* status) {
  return __all_sync(0xFFFFFFFFu, x_wait(bar, parity, dead, status));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Shared-memory matrix descriptor without swizzle: start address, leading and stride byte offsets
// in 16-byte units, descriptor version 1.
__device__ __forceinline__ uint64_t x_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo, uint32_t layout = 0) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46) |
         ((uint64_t)layout << 61);
}
// K-major operand with 128-byte swizzle: rows of 128 bytes, groups of 8 rows 1024 bytes apart (the leading offset is not used)
__device__ __forceinline__ uint64_t x_desc_rows(uint32_t saddr) { return x_desc(saddr, 16, 1024, 2); }
// One box of a 3-D tensor map (dims, keys, sequence x KV head) into shared memory; completion is
// counted in bytes on the mbarrier.
__device__ __forceinline__ void x_tma_box(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
__device__ __forceinline__ void x_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void x_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// The same, called by a whole converged warp: one elected lane issues. Loops around them stay uniform, so that the
// descriptors are formed by the scalar unit and need no transfer to it.
__device__ __forceinline__ void w_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, q;\nelect.sync _|q, 0xFFFFFFFF;\nsetp.ne.b32 p, %4, 0;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// The same with the A operand in tensor memory (row i of A in lane i, two fp16 values per column)
__device__ __forceinline__ void w_mma_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, q;\nelect.sync _|q, 0xFFFFFFFF;\nsetp.ne.b32 p, %4, 0;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// Four of them, issued by one elected lane: operands of the next K step lie STEP_A and STEP_B descriptor units (16 bytes) further.
template <int STEP_A, int STEP_B>
__device__ __forceinline__ void w_mma4(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, q, t;\n.reg .b64 a1, b1, a2, b2, a3, b3;\n"
      "add.u64 a1, %1, %5;\nadd.u64 b1, %2, %6;\nadd.u64 a2, %1, %7;\nadd.u64 b2, %2, %8;\nadd.u64 a3, %1, %9;\nadd.u64 b3, %2, %10;\n"
      "setp.ne.b32 p, %4, 0;\nsetp.eq.b32 t, 0, 0;\nelect.sync _|q, 0xFFFFFFFF;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %3, t;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, %3, t;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a3, b3, %3, t;\n}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "n"(STEP_A), "n"(STEP_B), "n"(2 * STEP_A), "n"(2 * STEP_B),
        "n"(3 * STEP_A), "n"(3 * STEP_B) : "memory");
}
// The same with A in tensor memory, COLS_A columns per K step
template <int COLS_A, int STEP_B>
__device__ __forceinline__ void w_mma4_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, q, t;\n.reg .b64 b1, b2, b3;\n.reg .b32 a1, a2, a3;\n"
      "add.u32 a1, %1, %5;\nadd.u64 b1, %2, %6;\nadd.u32 a2, %1, %7;\nadd.u64 b2, %2, %8;\nadd.u32 a3, %1, %9;\nadd.u64 b3, %2, %10;\n"
      "setp.ne.b32 p, %4, 0;\nsetp.eq.b32 t, 0, 0;\nelect.sync _|q, 0xFFFFFFFF;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, t;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, t;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, t;\n}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "n"(COLS_A), "n"(STEP_B), "n"(2 * COLS_A), "n"(2 * STEP_B),
        "n"(3 * COLS_A), "n"(3 * STEP_B) : "memory");
}
__device__ __forceinline__ void w_commit(uint32_t bar) {
  asm volatile(
      "{\n.reg .pred q;\nelect.sync _|q, 0xFFFFFFFF;\n"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}"
      ::"r"(bar) : "memory");
}
__device__ __forceinline__ void x_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void x_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
        "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
        "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
// 16 lanes x 64 columns: v[4 i + e] of lane l is row l / 4 + 8 (e / 2), column 8 i + 2 (l % 4) + e % 2
__device__ __forceinline__ void x_ld16x256(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void x_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
// 2^x, flushing denormals (2^-inf = 0)
__device__ __forceinline__ float x_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Byte offset of the 16-byte chunk `chunk` (8 K elements) of row `row` in a K-major operand whose K
// extent is `kchunks` chunks: core matrices of a row group side by side along K, row groups behind.
__device__ __forceinline__ uint32_t x_kmajor(int row, int chunk, int kchunks) {
  return (uint32_t)((row >> 3) * (kchunks * 128) + chunk * 128 + (row & 7) * 16);
}
// One box of a 2-D tensor map
__device__ __forceinline__ void x_tma_box2(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// The way out after a give-up: waits (bounded, whatever the flag says) for work this CTA has in flight, so that
// neither copies into its shared memory nor products into its TMEM outlive it.
__device__ __forceinline__ void x_drain(uint32_t bar, uint32_t parity) {
  for (int it = 0; it < (1 << 20); ++it) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return;
  }
}
__device__ __forceinline__ void x_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr) : "memory");
}

// ---- CTA pairs (clusters of two, the even CTA issues)
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// x_tma_box2 into the own CTA, counted on a barrier of either CTA of the pair (`bar`: cluster_addr)
__device__ __forceinline__ void pair_tma_box2(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// Arrives on the barrier at the same place in CTA `rank` of the cluster. What the arrival announces was written by the async
// proxy or fenced towards it, so no release at cluster scope is asked for (it takes most of a microsecond and would be paid per stage).
__device__ __forceinline__ void cluster_arrive(uint32_t bar, uint32_t rank) {
  asm volatile(
      "{\n.reg .b32 r;\nmapa.shared::cluster.u32 r, %0, %1;\n"
      "mbarrier.arrive.shared::cluster.b64 _, [r];\n}"
      ::"r"(bar), "r"(rank) : "memory");
}
// One whole warp of either CTA takes and returns the columns; the address goes to `slot` of the own CTA.
__device__ __forceinline__ void pair_tmem_alloc(uint32_t slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_tmem_free(uint32_t tmem, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}
// Four MMAs, K steps of 16 values whose operands lie STEP x 16 bytes apart (both K-major). M = 256 over the pair:
// either CTA holds 128 rows of A and half of the rows of B at the same shared-memory addresses, and all N columns of its 128 rows
// of D at the same TMEM address. Called by a converged warp of the even CTA; one elected lane issues them all (an election per
// instruction took longer than the MMAs).
template <int STEP>
__device__ __forceinline__ void pair_mma4(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, q, t;\n.reg .b64 a1, b1, a2, b2, a3, b3;\n"
      "add.u64 a1, %1, %5;\nadd.u64 b1, %2, %5;\nadd.u64 a2, %1, %6;\nadd.u64 b2, %2, %6;\nadd.u64 a3, %1, %7;\nadd.u64 b3, %2, %7;\n"
      "setp.ne.b32 p, %4, 0;\nsetp.eq.b32 t, 0, 0;\nelect.sync _|q, 0xFFFFFFFF;\n"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a1, b1, %3, t;\n"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a2, b2, %3, t;\n"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a3, b3, %3, t;\n}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "n"(STEP), "n"(2 * STEP), "n"(3 * STEP) : "memory");
}
// One poll of a barrier's phase; the answer may be asked for later
__device__ __forceinline__ uint32_t x_poll(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok;
}
// Arrives on the barrier at this address in both CTAs when the MMAs issued so far are done.
__device__ __forceinline__ void pair_commit(uint32_t bar) {
  asm volatile(
      "{\n.reg .pred q;\nelect.sync _|q, 0xFFFFFFFF;\n"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n}"
      ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// 16 lanes x 32 columns, laid out as x_ld16x256
__device__ __forceinline__ void x_ld16x256_32(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr) : "memory");
}

}  // namespace

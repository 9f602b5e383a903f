// tcgen05 (5th-generation tensor core) helpers for sm_100a, for CTAs in pairs (cta_group::2): tensor-memory allocation, shared-memory
// matrix descriptors for K-major 128-byte-swizzled f16 tiles, MMAs with A in tensor memory, commit, stores and loads of tensor memory.
// No copy here multicasts (a commit arrives on the barriers of both CTAs).
#pragma once
#include "common.cuh"

namespace infr {
namespace umma {

// ---- the pair -----------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t pair_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// One arrival on `bar` of the pair's first CTA.  What it tells of is in tensor memory and complete, ordered by tcgen05's own fences, so it
// orders no other memory of the pair.
__device__ __forceinline__ void arrive_first(uint64_t* bar) {
  asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %0, 0;\n\tmbarrier.arrive.shared::cluster.b64 _, [ra];\n\t}"
               ::"r"(smem_u32(bar)) : "memory");
}

// One lane of a converged warp.  Branching on this (and not on a lane number), in a branch the compiler knows to be
// warp-uniform, keeps the MMA operands in uniform registers: 9 cycles per tcgen05.mma against 55 from `if (lane == 0)`.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
  return p != 0;
}

// ---- tensor memory ------------------------------------------------------------------------------
// All 512 columns of both CTAs' tensor memory; one warp of each takes part.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* slot) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(slot)) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(taddr) : "memory");
}

__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Generic-proxy writes to shared memory (st.shared) become visible to the tensor core's reads.
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---- operand tiles in shared memory -------------------------------------------------------------
// A K-major tile of `rows` x 64 f16 (128 bytes per row), 128-byte swizzle: row r lives at byte
// r*128, its 16-byte chunk c at chunk position c ^ (r & 7).  Eight rows form one 1024-byte
// swizzle atom; the tile base must be 1024-byte aligned.

// 64-bit matrix descriptor for such a tile (start address, leading/stride byte offsets in units
// of 16 bytes, descriptor version 1, swizzle mode 128B).  `k16` selects the 16-element K slice
// inside the 64-element row (32 bytes each).
__device__ __forceinline__ uint64_t smem_desc_k_major_swz128(const void* tile, int k16) {
  const uint32_t addr = smem_u32(tile) + (uint32_t)k16 * 32u;
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);        // bits  0-13: start address
  d |= (uint64_t)1 << 16;                          // bits 16-29: leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024u >> 4) << 32;               // bits 32-45: stride byte offset = 8 rows * 128 B
  d |= (uint64_t)1 << 46;                          // bits 46-47: descriptor version (sm_100)
  d |= (uint64_t)2 << 61;                          // bits 61-63: swizzle mode 128 B
  return d;
}

// 32-bit instruction descriptor for kind::f16: f16 x f16 -> f32, both operands K-major.
__device__ __forceinline__ uint32_t idesc_f16_f32(int m, int n) {
  uint32_t d = 0;
  d |= 1u << 4;                      // D format: f32
  d |= 0u << 7;                      // A format: f16
  d |= 0u << 10;                     // B format: f16
  d |= 0u << 15;                     // A major: K
  d |= 0u << 16;                     // B major: K
  d |= (uint32_t)(n >> 3) << 17;     // N / 8
  d |= (uint32_t)(m >> 4) << 24;     // M / 16
  return d;
}

// D[tmem] (+)= A[tmem] * B[smem]^T for one K = 16 slice; A: lane = row, a 32-bit column = two K elements.  A and D: 128 rows in
// each CTA of the pair, at the same columns; B: half of the rows (tokens) in each, at the same place of shared memory.
__device__ __forceinline__ void mma_f16_ta(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(acc)
      : "memory");
}
// All MMAs issued so far by this thread arrive on `bar` of both CTAs when they have completed.
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

// 32 registers of every lane -> 32 consecutive columns of the lane's row (warp w: lanes 32 (w % 4) ..).
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n\t"
      "tcgen05.wait::st.sync.aligned;"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
        "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
        "r"(r[30]), "r"(r[31])
      : "memory");
}

// 16 accumulator rows (lanes) x 16 columns at each of four addresses as 8x8 fragments: thread T holds of row T / 4 (v[0],
// v[1]) and row T / 4 + 8 (v[2], v[3]) the columns 2 (T % 4), + 1; v[4..7] the same of the columns 8 further on.
__device__ __forceinline__ void tmem_ld_16x16_quad(uint32_t ta, uint32_t tb, uint32_t tc, uint32_t td, float (&a)[8], float (&b)[8], float (&c)[8],
                                                   float (&d)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%33];\n\t"
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%34];\n\t"
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%24,%25,%26,%27,%28,%29,%30,%31}, [%35];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=f"(a[0]), "=f"(a[1]), "=f"(a[2]), "=f"(a[3]), "=f"(a[4]), "=f"(a[5]), "=f"(a[6]), "=f"(a[7]), "=f"(b[0]), "=f"(b[1]), "=f"(b[2]),
        "=f"(b[3]), "=f"(b[4]), "=f"(b[5]), "=f"(b[6]), "=f"(b[7]), "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]), "=f"(c[4]), "=f"(c[5]),
        "=f"(c[6]), "=f"(c[7]), "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]), "=f"(d[4]), "=f"(d[5]), "=f"(d[6]), "=f"(d[7])
      : "r"(ta), "r"(tb), "r"(tc), "r"(td)
      : "memory");
}

}  // namespace umma
}  // namespace infr

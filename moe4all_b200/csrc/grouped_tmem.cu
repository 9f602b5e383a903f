// Grouped expert GEMMs on the 5th-generation tensor cores with the unpacked weights in tensor memory.
//
// Same contract as the mma.sync kernels of grouped_ffn.cu (reference: CPU stages B-D
// crates/infr-cpu/src/lib.rs:4051-4266; Vulkan native_gemm_mmq_q4k/q6k.comp): per expert segment
//   act = silu(Wg x) * (Wu x)      (MODE 0, k_wt_gemm<0, ...>)
//   y   = Wd act                   (MODE 1, k_wt_gemm<1, ...>)
//
// What such a GEMM pays for is the unpacking: every tile has to turn its blocks into f16 operands, whatever the number
// of tokens behind them, and the operand then crosses shared memory twice (written by the producers, read by the
// MMAs).  So the weights are the A operand and A lives in tensor memory: a producer thread owns one weight row, unpacks
// 64 of its weights into 32 registers and stores them with one tcgen05.st into its lane - no swizzle, no shared-memory
// traffic, no proxy fence.  The tokens are the B operand (N = the tile's tokens rounded up to 32, at most 160): the
// eight MMAs of a step take 640 cycles at 160 tokens, but 510 - 540 from 128 down, the time of reading A.  Tensor memory:
// two accumulators of 160 columns (gate and up rows, or the two halves of 256 output features) and three A stages of 64 columns
// (64 K elements of 256 rows).
//
// One persistent pair of CTAs per two SMs walks the jobs (tile, 2 x 256 weight rows, 256 of them in each CTA), tiles listed
// heaviest first and dealt out in a snake.  The MMAs are the pair's (cta_group::2, M 256): each CTA unpacks its own rows into its
// own tensor memory and brings half of the tile's tokens, and the tensor cores read both halves.  What it gives, with the Q6_K copies below
// (us cold and serialised, gate/up / down, one CTA by itself -> now): 777 tokens 60.5 / 58.8 -> 55.2 / 43.6, 4096 191 / 181 -> 164 / 139,
// 8192 of 28 MB experts 4058 / 3406 -> 3870 / 2346.  Two things were in the way: the 16-byte asynchronous copies of the gathered
// tokens (all their writes, not their latency: 20 KB a step, one copy instead of twenty a lane 177 -> 151; in a pair it is 10),
// and the MMAs, which take 640 cycles of eight at 160 tokens in pairs and 740 - 790 in one CTA with a wait for a stage between them.
// What it costs: 0.8 us a kernel (the cluster's two barriers, the paired allocation) and 500 - 1500 cycles a job, so calls of light tiles
// alone whose banks have no other gain are slower (4 - 64 rows of Q8_0 or Q4_K down banks 2 - 4 %, 256-wide experts 3 us of 53).
// Warp roles (24 warps of each CTA):
//   0-15   producers, two groups of eight on alternate K steps; afterwards they drain the accumulators
//   16     first CTA: issues the MMAs (one elected lane); second, gate/up: passes on that its tokens are there
//   then   token loaders: gate/up - four warps bring rows of the f16 token matrix straight from where the tokens are
//          (cp.async), two of them per K step; down - one warp, tiled copies of the tile's activations, 16 rows each, which
//          both CTAs count on the first one's barriers
//   last   raw-block loaders: 256 weights of 256 rows at a time, into a ring: Q4_K, Q5_K, Q8_0 and the down banks' Q6_K by
//          tiled copies, which one warp requests (gate/up: two more pass tokens on), other formats word by word with cp.async
//          (rows on an odd word pitch, free of bank conflicts)
// All rings run on across jobs; every wait on a barrier of shared memory is bounded (the cluster's two barriers and the paired allocation
// have no limit of their own: nothing that either CTA does ahead of them waits for long).
//
// Reading out a full tile of the down kernel takes 5100 cycles beside the 7700 of its K loop at 512 inputs, with the tensor cores
// idle: there is one set of accumulators.
// Down with Q6_K, whose blocks are 210 bytes: as words by cp.async the copies were what everything waited for (without them 3704 ->
// 2104 us, 8192 tokens of 28 MB experts).  Now a tiled copy brings the 240 bytes around a block, of one row in every 1, 2, 4 or 8
// (row_shift), so that a warp's rows have one offset inside them: 3704 -> 2526 us, 4096 tokens of 2 MB experts 177 -> 142.
#include <cuda.h>

#include <algorithm>

#include "formats.cuh"
#include "kernels.cuh"
#include "umma.cuh"
#include "tma.cuh"

namespace infr {
namespace {

using namespace umma;

constexpr int WN = 160;              // most tokens of a tile
constexpr int WR = 256;              // weight rows of a job
constexpr int W_PRODUCERS = 512;
constexpr int W_THREADS = 768;
constexpr int W_MMA_WARP = 16, W_TOK_WARP = 17;
__host__ __device__ constexpr int wt_tok_warps(int mode) { return mode == 0 ? 4 : 1; }
__host__ __device__ constexpr int wt_raw_warp(int mode) { return W_TOK_WARP + wt_tok_warps(mode); }
__host__ __device__ constexpr int wt_raw_warps(int mode) { return mode == 0 ? 3 : 4; }

// Q4_K, Q5_K, Q8_0 (both roles): tiled copies, rows of whole 16-byte pieces.  Q6_K (down): tiled copies of the 240 bytes around a
// block of 210, over 2^row_shift rows at a time, whose bytes are whole 16-byte pieces.  Any: words, on an odd word pitch.
enum WtFormat { WT_Q4K, WT_Q5K, WT_Q80, WT_Q6K, WT_ANY };
__host__ __device__ constexpr bool wt_tiled(int fmt) { return fmt <= WT_Q6K; }
constexpr uint32_t W_Q6K_BOX = 240;  // 15 pieces of 16 bytes: 14 bytes of offset and 210 of block, rounded up; odd, so that eight
                                     // rows' pieces are in different banks

// Warps of the second CTA that pass its gate/up tokens on (relay_tokens).
__host__ __device__ constexpr int wt_relays(int mode, int fmt) { return mode == 0 ? (wt_tiled(fmt) ? 3 : 1) : 0; }
// Stages of the token ring.  Gate/up of Q4_K and Q5_K: as many as leave room for two raw stages, over which the hand-over's time (relay_tokens)
// is spread (six and four of Q4_K -> ten and two: 777 tokens 176 -> 170 us the call, 4096 482 -> 474; Q5_K level); Q8_0's raw stages leave
// room for six, and words need no more (MXFP4 840 either way).  Down: six (four 2 - 3 % slower, eight level).
__host__ __device__ constexpr int wt_b_stages(int mode, int fmt) { return mode == 0 && (fmt == WT_Q4K || fmt == WT_Q5K) ? 10 : 6; }
constexpr int W_MAX_B_STAGES = 10;
constexpr uint32_t W_B_STAGE = WN / 2 * 128;   // 64 K elements of half of the tile's tokens
constexpr uint32_t W_PATCH = 1280;             // per warp: 16 rows x 80 B (f16) or 8 rows x 144 B (f32)
constexpr int W_MAX_RAW = 4;
constexpr int W_A_STAGES = 3;
constexpr uint32_t W_A_COL = 2 * WN;           // first A column of tensor memory
constexpr float W_PRESCALE = 256.0f;           // keeps block scales out of the f16 subnormals
constexpr float W_POSTSCALE = 1.0f / 256.0f;

__device__ __forceinline__ uint32_t h2_as_u32(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 u32_as_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
__device__ __forceinline__ __half2 h2_const(uint32_t bits) { return u32_as_h2(bits | (bits << 16)); }

// ---- copy forms only this file uses -------------------------------------------------------------------

// One arrival on the first CTA's barriers of ring positions i .. i + PER - 1, for what threads wrote to this CTA's shared memory: released at
// the scope of the pair, acquired there by pair_wait.
template <int PER, int STAGES>
__device__ __forceinline__ void release_first(uint64_t* ring, int i) {
  asm volatile("fence.acq_rel.cluster;" ::: "memory");
#pragma unroll
  for (int k = 0; k < PER; ++k)
    asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %0, 0;\n\tmbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [ra];\n\t}"
                 ::"r"(smem_u32(&ring[(i + k) % STAGES])) : "memory");
}
// One tiled copy into this CTA's shared memory, counted in bytes on `bar` of the pair's first CTA.
__device__ __forceinline__ void tma_load_2d_first(void* smem_dst, const CUtensorMap* tm, int x, int y, uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %2, 0;\n\t"
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4}], [ra];\n\t}"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_u32(bar)), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
// One arrival on `bar` once all copies this thread has issued so far are there.
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Bounded wait of these kernels: a look, then waits that the hardware suspends (spinning warps took a third of the issue
// slots from the producers).  The limit is a few seconds.
#define WT_WAIT(NAME, SCOPE)                                                                                                                     \
  __device__ __forceinline__ bool NAME(uint64_t* bar, uint32_t parity) {                                                                         \
    uint32_t ok;                                                                                                                                 \
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.acquire." SCOPE ".shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"    \
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");                                                                        \
    if (ok) return true;                                                                                                                         \
    for (uint32_t i = 0; i < (1u << 21); ++i) {                                                                                                  \
      asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire." SCOPE ".shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}" \
                   : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(1000u) : "memory");                                                          \
      if (ok) return true;                                                                                                                       \
    }                                                                                                                                            \
    return false;                                                                                                                                \
  }
WT_WAIT(wt_wait, "cta")
WT_WAIT(pair_wait, "cluster")  // acquires what release_first released
#undef WT_WAIT

// Meeting of the four warps behind `bar` (bounded, unlike the barriers of the CTA).
__device__ __forceinline__ bool meet(uint64_t* bar, uint32_t& phase) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
  const bool ok = __all_sync(0xFFFFFFFFu, wt_wait(bar, phase));
  phase ^= 1;
  return ok;
}

// ---- unpacking: 64 weights of a row -> 32 columns, K order 0,2,1,3 inside every four ---------------------
//
// Codes become f16 by setting the exponent bits of 1024 (or 64 for codes that sit four bits up) above them, the
// offset comes off exactly, and scale and min are applied by one multiply-add.

// Scales of two groups, given as bytes 0 and 1 of `pair` (at most 63): d * code, both rounded once.
__device__ __forceinline__ __half2 scale_pair(uint32_t pair, __half2 d) {
  return __hmul2(__hsub2(u32_as_h2(__byte_perm(pair, 0x64u, 0x4140)), h2_const(0x6400u)), d);
}

// Step j of a Q4_K block; the row starts on a 16-byte boundary.
__device__ __forceinline__ void unpack_q4k(const unsigned char* row, int j, uint32_t (&o)[32]) {
  const uint4 hd = *reinterpret_cast<const uint4*>(row);
  const uint4 qa = *reinterpret_cast<const uint4*>(row + 16 + 32 * j), qb = *reinterpret_cast<const uint4*>(row + 32 + 32 * j);
  uint32_t scp, mp;
  q4k_scale_min_pair(hd.y, hd.z, hd.w, j, scp, mp);
  const __half2 dd = __hmul2(u32_as_h2(hd.x ^ 0x80000000u), h2_const(0x5C00u));  // 256 (d, -dmin)
  const __half2 s2 = scale_pair(scp, __low2half2(dd)), m2 = scale_pair(mp, __high2half2(dd));
  const __half2 sl = __low2half2(s2), sh = __high2half2(s2), ml = __low2half2(m2), mh = __high2half2(m2);
  const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t v = w[i] >> 8;
    const __half2 l02 = __hsub2(u32_as_h2((w[i] & 0x000F000Fu) | 0x64006400u), h2_const(0x6400u));
    const __half2 l13 = __hsub2(u32_as_h2((v & 0x000F000Fu) | 0x64006400u), h2_const(0x6400u));
    const __half2 h02 = __hsub2(u32_as_h2((w[i] & 0x00F000F0u) | 0x54005400u), h2_const(0x5400u));
    const __half2 h13 = __hsub2(u32_as_h2((v & 0x00F000F0u) | 0x54005400u), h2_const(0x5400u));
    o[2 * i] = h2_as_u32(__hfma2(l02, sl, ml));
    o[2 * i + 1] = h2_as_u32(__hfma2(l13, sl, ml));
    o[16 + 2 * i] = h2_as_u32(__hfma2(h02, sh, mh));
    o[16 + 2 * i + 1] = h2_as_u32(__hfma2(h13, sh, mh));
  }
}

// Four signed bytes with one scale: 1024 + (byte + 128) in one operation (the sign bit flips with the exponent's bits), the
// offset off exactly, times s.
__device__ __forceinline__ void codes4_mul(uint32_t c, __half2 s, uint32_t& o02, uint32_t& o13) {
  o02 = h2_as_u32(__hmul2(__hsub2(u32_as_h2((c & 0x00FF00FFu) ^ 0x64806480u), h2_const(0x6480u)), s));
  o13 = h2_as_u32(__hmul2(__hsub2(u32_as_h2(((c >> 8) & 0x00FF00FFu) ^ 0x64806480u), h2_const(0x6480u)), s));
}

// Two int8 scales (bytes of `w` picked by the selector) times d: exact integers in f16, one rounding.
__device__ __forceinline__ __half2 i8_scale_pair(uint32_t w, uint32_t sel, __half2 d) {
  return __hmul2(__hsub2(u32_as_h2(__byte_perm(w ^ 0x80808080u, 0x64u, sel)), h2_const(0x6480u)), d);
}

// Step 2 h + g of a Q6_K block; the block starts `mis` (0 or 16) bits into the first word of `row`.
__device__ __forceinline__ void unpack_q6k(const uint32_t* row, int mis, int h, int g, uint32_t (&o)[32]) {
  auto word = [&](int i) { return __funnelshift_r(row[i], row[i + 1], mis); };
  const uint32_t sc = word(48 + 2 * h + g);  // scales of the step's four groups of 16
  const __half2 d = __hmul2(u32_as_h2(__byte_perm(row[52] >> mis, 0u, 0x1010)), h2_const(0x5C00u));  // f16 d: bytes 208, 209
  const __half2 s01 = i8_scale_pair(sc, 0x4140, d), s23 = i8_scale_pair(sc, 0x4342, d);
  uint32_t hq[8];
  {
    uint32_t a = row[32 + 8 * h];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t b = row[33 + 8 * h + i];
      hq[i] = __funnelshift_r(a, b, mis);
      a = b;
    }
  }
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    const int rot = (4 - 4 * g - 2 * part) & 31;  // brings bits 2 qd, 2 qd + 1 of a byte to its bits 4, 5
    const __half2 s_a = __low2half2(part ? s23 : s01), s_b = __high2half2(part ? s23 : s01);
    uint32_t a = row[16 * h + 8 * part];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t b = row[16 * h + 8 * part + 1 + i];
      const uint32_t L = __funnelshift_r(a, b, mis + 4 * g), H = __funnelshift_l(hq[i], hq[i], rot);
      a = b;
      const uint32_t c = (H & 0x30303030u) | (L & 0x0F0F0F0Fu);
      const uint32_t c02 = __byte_perm(c, 0x64u, 0x4240), c13 = __byte_perm(c, 0x64u, 0x4341);
      const __half2 s = i < 4 ? s_a : s_b;
      o[16 * part + 2 * i] = h2_as_u32(__hmul2(__hsub2(u32_as_h2(c02), h2_const(0x6420u)), s));
      o[16 * part + 2 * i + 1] = h2_as_u32(__hmul2(__hsub2(u32_as_h2(c13), h2_const(0x6420u)), s));
    }
  }
}

// Half h (128 weights, two steps) of a Q6_K block in 16-byte pieces, words realigned: the block starts WO words and `mis` (0 or 16)
// bits into the 16-byte boundary `row`.
struct Q6kHalf {
  uint32_t ql[16], qh[8], sc[2], d;
};
template <int WO>
__device__ __forceinline__ void fetch_q6k_half(const unsigned char* row, int h, int mis, Q6kHalf& r) {
  {
    uint32_t v[20];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const uint4 x = *reinterpret_cast<const uint4*>(row + 64 * h + 16 * i);
      v[4 * i] = x.x, v[4 * i + 1] = x.y, v[4 * i + 2] = x.z, v[4 * i + 3] = x.w;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) r.ql[i] = __funnelshift_r(v[WO + i], v[WO + i + 1], mis);
  }
  {
    uint32_t v[12];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const uint4 x = *reinterpret_cast<const uint4*>(row + 128 + 32 * h + 16 * i);
      v[4 * i] = x.x, v[4 * i + 1] = x.y, v[4 * i + 2] = x.z, v[4 * i + 3] = x.w;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) r.qh[i] = __funnelshift_r(v[WO + i], v[WO + i + 1], mis);
  }
  const uint4 a = *reinterpret_cast<const uint4*>(row + 192), b = *reinterpret_cast<const uint4*>(row + 208);
  const uint32_t v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  const uint32_t s0 = h ? v[WO + 2] : v[WO], s1 = h ? v[WO + 3] : v[WO + 1], s2 = h ? v[WO + 4] : v[WO + 2];
  r.sc[0] = __funnelshift_r(s0, s1, mis);
  r.sc[1] = __funnelshift_r(s1, s2, mis);
  r.d = v[WO + 4] >> mis;
}

// Step 2 h + G from the half.
template <int G>
__device__ __forceinline__ void unpack_q6k_half(const Q6kHalf& r, uint32_t (&o)[32]) {
  const __half2 d = __hmul2(u32_as_h2(__byte_perm(r.d, 0u, 0x1010)), h2_const(0x5C00u));
  const __half2 s01 = i8_scale_pair(r.sc[G], 0x4140, d), s23 = i8_scale_pair(r.sc[G], 0x4342, d);
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    const __half2 s_a = __low2half2(part ? s23 : s01), s_b = __high2half2(part ? s23 : s01);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t L = G ? r.ql[8 * part + i] >> 4 : r.ql[8 * part + i];
      const uint32_t H = G ? (part ? r.qh[i] >> 2 : r.qh[i]) : (part ? r.qh[i] << 2 : r.qh[i] << 4);  // the code's bits 4, 5 in place
      const uint32_t c = (H & 0x30303030u) | (L & 0x0F0F0F0Fu);
      const uint32_t c02 = __byte_perm(c, 0x64u, 0x4240), c13 = __byte_perm(c, 0x64u, 0x4341);
      const __half2 s = i < 4 ? s_a : s_b;
      o[16 * part + 2 * i] = h2_as_u32(__hmul2(__hsub2(u32_as_h2(c02), h2_const(0x6420u)), s));
      o[16 * part + 2 * i + 1] = h2_as_u32(__hmul2(__hsub2(u32_as_h2(c13), h2_const(0x6420u)), s));
    }
  }
}

// A step of eight Q8_0 blocks: 68 bytes = two blocks, the first on a word boundary, the second two bytes past one.
// w(i): word i of the step.
template <typename Word>
__device__ __forceinline__ void unpack_q80(Word w, uint32_t (&o)[32]) {
  const uint32_t mid = w(8);
  const __half2 d = __hmul2(u32_as_h2(__byte_perm(w(0), mid, 0x7610)), h2_const(0x5C00u));
#pragma unroll
  for (int i = 0; i < 8; ++i) codes4_mul(__funnelshift_r(w(i), w(i + 1), 16), __low2half2(d), o[2 * i], o[2 * i + 1]);
#pragma unroll
  for (int i = 0; i < 8; ++i) codes4_mul(w(9 + i), __high2half2(d), o[16 + 2 * i], o[16 + 2 * i + 1]);
}
// The row on a 16-byte boundary: the words of step J are words J .. J + 16 of five 16-byte pieces.
template <int J>
__device__ __forceinline__ void unpack_q80_row(const unsigned char* row, uint32_t (&o)[32]) {
  uint32_t v[20];
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const uint4 x = *reinterpret_cast<const uint4*>(row + 64 * J + 16 * i);
    v[4 * i] = x.x, v[4 * i + 1] = x.y, v[4 * i + 2] = x.z, v[4 * i + 3] = x.w;
  }
  unpack_q80([&](int i) { return v[J + i]; }, o);
}

// Step j of a Q5_K (FIVE) or Q4_K block.  hd, qh: the block's first 16 bytes and its high bits; qs(i): code word i of the step.
template <bool FIVE, typename Word>
__device__ __forceinline__ void unpack_k45(const uint4& hd, const uint32_t (&qh)[8], Word qs, int j, uint32_t (&o)[32]) {
  uint32_t scp, mp;
  q4k_scale_min_pair(hd.y, hd.z, hd.w, j, scp, mp);
  const __half2 dd = __hmul2(u32_as_h2(hd.x ^ 0x80000000u), h2_const(0x5C00u));
  const __half2 s2 = scale_pair(scp, __low2half2(dd)), m2 = scale_pair(mp, __high2half2(dd));
  const __half2 sl = __low2half2(s2), sh = __high2half2(s2), ml = __low2half2(m2), mh = __high2half2(m2);
  const int rl = (4 - 2 * j) & 31, rh = (3 - 2 * j) & 31;  // brings bit 2 j (2 j + 1) of a byte to its bit 4
  constexpr uint32_t B4 = FIVE ? 0x00100010u : 0u;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t w = qs(i), q = FIVE ? qh[i] : 0u;
    const uint32_t bl = __funnelshift_l(q, q, rl), bh = __funnelshift_l(q, q, rh), wh = w >> 4;
    const uint32_t l02 = (bl & B4) | ((w & 0x000F000Fu) | 0x64006400u), l13 = ((bl >> 8) & B4) | (((w >> 8) & 0x000F000Fu) | 0x64006400u);
    const uint32_t h02 = (bh & B4) | ((wh & 0x000F000Fu) | 0x64006400u), h13 = ((bh >> 8) & B4) | (((wh >> 8) & 0x000F000Fu) | 0x64006400u);
    o[2 * i] = h2_as_u32(__hfma2(__hsub2(u32_as_h2(l02), h2_const(0x6400u)), sl, ml));
    o[2 * i + 1] = h2_as_u32(__hfma2(__hsub2(u32_as_h2(l13), h2_const(0x6400u)), sl, ml));
    o[16 + 2 * i] = h2_as_u32(__hfma2(__hsub2(u32_as_h2(h02), h2_const(0x6400u)), sh, mh));
    o[16 + 2 * i + 1] = h2_as_u32(__hfma2(__hsub2(u32_as_h2(h13), h2_const(0x6400u)), sh, mh));
  }
}
// Word by word (any word boundary), and in 16-byte pieces.
template <bool FIVE>
__device__ __forceinline__ void unpack_k45_words(const uint32_t* row, int j, uint32_t (&o)[32]) {
  uint32_t qh[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) qh[i] = FIVE ? row[4 + i] : 0u;
  unpack_k45<FIVE>(make_uint4(row[0], row[1], row[2], row[3]), qh, [&](int i) { return row[(FIVE ? 12 : 4) + 8 * j + i]; }, j, o);
}
__device__ __forceinline__ void unpack_q5k_row(const unsigned char* row, int j, uint32_t (&o)[32]) {
  const uint4 ha = *reinterpret_cast<const uint4*>(row + 16), hb = *reinterpret_cast<const uint4*>(row + 32);
  const uint4 qa = *reinterpret_cast<const uint4*>(row + 48 + 32 * j), qb = *reinterpret_cast<const uint4*>(row + 64 + 32 * j);
  const uint32_t qh[8] = {ha.x, ha.y, ha.z, ha.w, hb.x, hb.y, hb.z, hb.w}, q[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
  unpack_k45<true>(*reinterpret_cast<const uint4*>(row), qh, [&](int i) { return q[i]; }, j, o);
}

// Step j of 256 weights in any format, through the code view (`row`: a copy in shared memory, words aligned as in the bank).
__device__ __forceinline__ void unpack_codes(int dt, const unsigned char* row, int j, uint32_t (&o)[32]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t c[4];
    float A, B;
    int off;
    fmt_codes16<false>(dt, row, 4 * j + q, c, A, B, off);
    const __half2 a2 = __float2half2_rn(A * W_PRESCALE), b2 = __float2half2_rn(B * W_PRESCALE), o2 = __float2half2_rn((float)(1024 + off));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __half2 v02 = __hsub2(u32_as_h2((c[i] & 0x00FF00FFu) | 0x64006400u), o2), v13 = __hsub2(u32_as_h2(((c[i] >> 8) & 0x00FF00FFu) | 0x64006400u), o2);
      o[8 * q + 2 * i] = h2_as_u32(__hfma2(v02, a2, b2));
      o[8 * q + 2 * i + 1] = h2_as_u32(__hfma2(v13, a2, b2));
    }
  }
}

// ---- results ------------------------------------------------------------------------------------------

// Two f32 as f16, saturated to the largest finite value.
__device__ __forceinline__ uint32_t f16x2_sat(float a, float b) {
  uint32_t r;
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}

__device__ __forceinline__ float exp2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Out of line: the activations other than SiLU, and the clamp.
__device__ __noinline__ float gated_act_general(int act, float clamp, float g, float u) { return gated_act<true>(act, clamp, g, u); }

// Four outputs of the down kernel in 12 bytes: each keeps sign, exponent and 15 mantissa bits of its f32 (rounded to the
// nearest, within 2^-16 of itself), the upper 16 bits in `hi`, the last 8 in `lo`.  Every output has an exponent of its own:
// the outputs of a trained down projection differ by factors of hundreds to thousands from one feature to the next, and an
// exponent shared by four (14-bit mantissas, 8 bytes) left neighbours of an output 1000 times theirs with 5e-2 of themselves.
// A chunk of 4096 tokens, 2048 wide, eight experts of 256 and the shared one each: 560 us (8 bytes: 553; f32 rows: 573).
__device__ __forceinline__ void pack_y4(float a, float b, float c, float d, uint2& hi, uint32_t& lo) {
  uint32_t q[4] = {__float_as_uint(a), __float_as_uint(b), __float_as_uint(c), __float_as_uint(d)};
  // (sums of products of f16 stay below 2^50, so what is not finite is an infinity or the tensor core's NaN, 0x7FFFFFFF: the
  // first keeps its upper bits under the addition, the second by the limit)
#pragma unroll
  for (int i = 0; i < 4; ++i) q[i] = (uint32_t)(min((int)q[i], 0x7FFFFF7F) + 0x80);
  hi = make_uint2(__byte_perm(q[0], q[1], 0x7632), __byte_perm(q[2], q[3], 0x7632));
  lo = __byte_perm(__byte_perm(q[0], q[1], 0x0051), __byte_perm(q[2], q[3], 0x0051), 0x5410);
}

// ---- the kernel ---------------------------------------------------------------------------------------

struct WtBars {
  uint64_t full_a[W_A_STAGES], empty_a[W_A_STAGES];      // A stages in tensor memory
  uint64_t full_b[W_MAX_B_STAGES], empty_b[W_MAX_B_STAGES];  // token stages
  uint64_t full_raw[W_MAX_RAW], empty_raw[W_MAX_RAW];    // raw-block stages
  uint64_t done, drained;                                // accumulators complete / read
  uint64_t patch[4];                                     // down: the four warps of a set of tokens have their outputs in order
};

// Position in a ring of n stages, running on across jobs.
struct RingPos {
  int s = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void next(int n) {
    if (++s == n) {
      s = 0;
      phase ^= 1;
    }
  }
};

struct WtParams {
  GroupedParams g;
  int n_blk, n_pair;  // blocks of 256 weight rows per tile; pairs of them
  int k_blocks;     // 256-element blocks along K
  int rb;           // stages of the raw ring
  uint32_t raw_pitch, raw_stage;  // bytes per row and per stage
  int row_shift;            // down: producer warp w holds the rows (32 (w >> row_shift) + lane) 2^row_shift + w % 2^row_shift
  // gate/up tokens: row of the token matrix behind grouped row `pos`
  const int* pair_of_pos;   // null: the rows are grouped already
  const int* seg_off;       // [n_seg_routed] = grouped rows ahead of the shared expert's
  int n_seg_routed, n_used;
};

// Job i of this pair of CTAs: rounds of as many jobs as there are pairs, every other round dealt out backwards (the tiles' cost
// falls along the list).
__device__ __forceinline__ int wt_job(int i) {
  const int pairs = (int)gridDim.x >> 1, me = (int)blockIdx.x >> 1;
  return i * pairs + ((i & 1) ? pairs - 1 - me : me);
}
// Weight rows of a job that are this CTA's: block blk0 of 256, or, where the blocks (of a down bank) are odd in number and the last one is
// left to a pair by itself, half of it: 128 rows go through the first accumulator, the second and its producers rest.
// (Both CTAs doing all of it, us a call of 4096 tokens of Q4_K / Q6_K: 256 wide 122 -> 116, 768 wide 191 -> 187, of 2048-wide experts 438 -> 426;
// 512 tokens of Q4_K, 256 wide: 61 -> 59, one CTA by itself 55; 768 wide 91 -> 89, 88.)
struct JobBlock {
  int tile, blk0;
  bool lone;
};
__device__ __forceinline__ JobBlock wt_block(int job, int n_pair, int n_blk, int rank) {
  JobBlock j;
  j.tile = job / n_pair;
  const int b = 2 * (job - j.tile * n_pair);
  j.lone = b + 1 == n_blk;
  j.blk0 = j.lone ? b : b + rank;
  return j;
}

// The second CTA, gate/up: passes on to the first that its tokens are there, PER steps at a time, from step PER `first` of all its jobs' on
// PER `by` apart.  They are ordinary writes to shared memory (cp.async) that the MMAs of another CTA read, so they are released at the scope
// of the pair.  Such a release takes longer than a step of 800 cycles: one warp, a release a step, is what everything waits for (777 tokens
// 220 us the call, 1024 of Q8_0 251, 64 rows of 28 MB experts of Q8_0 2220).  Three warps 177, 208, 1440; and two steps a release 177, 208,
// 1399.  Formats that come word by word leave one warp, and their steps are longer: a release a step (48 rows of 28 MB experts of MXFP4
// 5640 us, two steps a release 5970).
template <int PER, int STAGES>
__device__ __forceinline__ bool relay_tokens(WtBars& bars, int n_jobs, int steps, int first, int by) {
  int n = 0;
  for (int it = 0; wt_job(it) < n_jobs; ++it) n += steps;  // a multiple of four
  for (int i = PER * first; i < n; i += PER * by) {
    for (int k = 0; k < PER; ++k)
      if (!__all_sync(0xFFFFFFFFu, wt_wait(&bars.full_b[(i + k) % STAGES], ((i + k) / STAGES) & 1))) return false;
    if (elect_one()) {
      fence_proxy_async();
      release_first<PER, STAGES>(bars.full_b, i);
    }
    __syncwarp();
  }
  return true;
}

// Lane of an operand tile -> weight row: gate/up rows go in the order 0,2,1,3 inside every four, so that the
// activations come out in the K order of the down kernel's operands.
__device__ __forceinline__ int wt_row_of_lane(int mode, int l) { return mode == 0 ? ((l & ~3) | ((l & 1) << 1) | ((l >> 1) & 1)) : l; }

// TRACED: with a trace buffer attached, the job of tile p.trace_tile over the first weight rows writes phase stamps.  Gate/up
// (down: 4 slots on): 40 the job's start, 41 its first raw blocks there, 42 accumulators complete, 43 drained.  Of its first 16
// K steps (down: 64 slots on): 64 + 4 i the first producer warp looks for the raw blocks of step 2 i, 65 + 4 i has them, 66 + 4 i
// has unpacked its weights, 67 + 4 i has stored them; 96 + 2 i the operands of step i are there, 97 + 2 i its MMAs are issued.
// A variant of its own: the plain one has neither the pointer's registers nor a branch per step.  ODD: the 256-row blocks are odd in number
// (down), a variant of its own too (in one kernel 4096 tokens of 2048 wide take 488 us a call, not 480).
template <int MODE, int FMT, bool TRACED, bool ODD>
__global__ void __launch_bounds__(W_THREADS, 1) k_wt_gemm(const __grid_constant__ WtParams w, const __grid_constant__ CUtensorMap tm_w0,
                                                         const __grid_constant__ CUtensorMap tm_w1, const __grid_constant__ CUtensorMap tm_s0,
                                                         const __grid_constant__ CUtensorMap tm_s1, const __grid_constant__ CUtensorMap tm_act) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) WtBars bars;
  __shared__ uint32_t s_tmem;
  constexpr int RAW_WARP = wt_raw_warp(MODE), RAW_WARPS = wt_raw_warps(MODE), RELAYS = wt_relays(MODE, FMT), PER = RELAYS > 1 ? 2 : 1, B_STAGES = wt_b_stages(MODE, FMT);
  const GroupedParams& p = w.g;
  unsigned char* b_ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* raw_ring = b_ring + B_STAGES * W_B_STAGE;
  unsigned char* patches = raw_ring + (size_t)w.rb * w.raw_stage;
  // (shuffles and votes mark what is the same in the whole warp: the MMA operands then stay in uniform registers)
  const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
  // Tiles and rows come from the kernels ahead in the stream.  The down kernel starts when the gate/up kernel already has them:
  // only its token copies wait (for the activations), its weights are on their way and unpacked by then.
  if (MODE == 0) pdl_wait();
  pdl_trigger();
  const int rank = __shfl_sync(0xFFFFFFFFu, (int)pair_rank(), 0);
  const int n_jobs = __shfl_sync(0xFFFFFFFFu, __ldcg(p.n_tiles) * w.n_pair, 0);
  if (wt_job(0) >= n_jobs) {
    if (MODE == 1) pdl_wait();
    return;
  }

  if (tid == 0) {
    for (int s = 0; s < W_A_STAGES; ++s) {
      mbar_init(&bars.full_a[s], 16);
      mbar_init(&bars.empty_a[s], 1);
    }
    for (int s = 0; s < B_STAGES; ++s) {
      mbar_init(&bars.full_b[s], MODE == 1 ? 1 : rank == 0 ? 65 : 64);
      mbar_init(&bars.empty_b[s], 1);
    }
    for (int s = 0; s < W_MAX_RAW; ++s) {
      mbar_init(&bars.full_raw[s], wt_tiled(FMT) ? 1 : RAW_WARPS * 32);
      mbar_init(&bars.empty_raw[s], W_PRODUCERS / 32);
    }
    mbar_init(&bars.done, 1);
    mbar_init(&bars.drained, 2 * W_PRODUCERS / 32);
    for (int s = 0; s < 4; ++s) mbar_init(&bars.patch[s], 4);
    mbar_fence_init();
  }
  if (warp == W_MMA_WARP) tmem_alloc_pair(&s_tmem);
  fence_before_sync();
  pair_sync();  // the other CTA's barriers are there, and both have their tensor memory
  fence_after_sync();
  // All 512 columns are this CTA's, so they start at column 0 of lane 0, and addresses below are constants.  Were it ever
  // otherwise, every role would leave at once and the call report it.
  constexpr uint32_t tmem = 0;
  const int kb = w.k_blocks;
  bool ok = s_tmem == tmem;

  if (warp < W_PRODUCERS / 32) {
    // ---- producers: unpack, then drain ----
    const int g = warp >> 3, role = (warp >> 2) & 1, q = warp & 3;
    const int dt = MODE == 1 ? p.down_dt : (role ? p.up_dt : p.gate_dt);
    const int half_word = (int)(row_bytes(dt, 256) & 2);  // blocks of an odd number of half-words: every other one is off a word boundary
    const uint32_t a_addr = tmem + ((uint32_t)(q * 32) << 16) + W_A_COL + 32u * role;
    unsigned char* patch = patches + (size_t)warp * W_PATCH;
    const uint32_t patch_u = smem_u32(patch);
    RingPos rp, ap;  // raw blocks; A stages
    if (g) ap.next(W_A_STAGES);
    if (g && FMT == WT_Q6K) ap.next(W_A_STAGES);
    uint32_t d_phase = 0, m_phase = 0;
    for (int it = 0; ok; ++it) {
      const int job = wt_job(it);
      if (job >= n_jobs) break;
      const JobBlock jb = wt_block(job, w.n_pair, w.n_blk, rank);
      const int tile = jb.tile, blk0 = jb.blk0;
      const bool lone = ODD && jb.lone;
      // row of the raw stage (down: the rows of a warp have one offset from the 16-byte boundary)
      const int w8 = (lone ? 4 * rank : 4 * role) + q, sub = w8 & ((1 << w.row_shift) - 1);
      const int slot = MODE == 0 ? role * 128 + wt_row_of_lane(MODE, q * 32 + lane)
                                 : (sub << (8 - w.row_shift)) + (w8 >> w.row_shift) * 32 + lane;
      const int e = __ldcg(p.tile_expert + tile), row0 = __ldcg(p.tile_row0 + tile), rows_valid = __ldcg(p.tile_rows + tile);
      const int wrow = MODE == 0 ? blk0 * 128 + (slot & 127) : blk0 * WR + slot;
      unsigned long long* tr = TRACED && tile == p.trace_tile && blk0 == 0 && rank == 0 ? p.trace : nullptr;
      if (TRACED) trace_stamp(tr, 40 + 4 * MODE);
      for (int blk = 0; blk < kb; ++blk) {
        if (TRACED && blk < 4) trace_stamp(tr, 64 + 64 * MODE + 8 * blk);
        if (!wt_wait(&bars.full_raw[rp.s], rp.phase)) { ok = false; break; }
        if (TRACED && blk == 0) trace_stamp(tr, 41 + 4 * MODE);
        if (TRACED && blk < 4) trace_stamp(tr, 65 + 64 * MODE + 8 * blk);
        if (lone && role) {  // nothing to unpack: only the arrivals that the barriers count
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars.empty_raw[rp.s]);
          for (int h = 0; h < 2 && ok; ++h) {
            ok = __all_sync(0xFFFFFFFFu, wt_wait(&bars.empty_a[ap.s], ap.phase ^ 1));
            if (ok && lane == 0) arrive_first(&bars.full_a[ap.s]);
            for (int i = FMT != WT_Q6K ? 2 : h ? 3 : 1; i > 0; --i) ap.next(W_A_STAGES);
          }
          if (!ok) break;
          rp.next(w.rb);
          continue;
        }
        const unsigned char* row = raw_ring + (size_t)rp.s * w.raw_stage + (size_t)slot * w.raw_pitch;
        const int mis = ((wrow * kb + blk) & 1) * half_word;  // bytes of the stage's first word ahead of the block
        Q6kHalf half;
        if (FMT == WT_Q6K) {
          // The group's two steps are one half of the block (the low and the high bits of the same code bytes), so its words are read
          // and realigned once for both, and the stage is free as soon as they are in registers.
          const int off = ((int)Q6K_BLOCK_BYTES * (sub * kb + blk)) & 15, bits = (off & 2) * 8;
          switch (off >> 2) {
            case 0: fetch_q6k_half<0>(row, g, bits, half); break;
            case 1: fetch_q6k_half<1>(row, g, bits, half); break;
            case 2: fetch_q6k_half<2>(row, g, bits, half); break;
            default: fetch_q6k_half<3>(row, g, bits, half); break;
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars.empty_raw[rp.s]);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t o[32];
          const int j = 2 * h + g;
          const uint32_t* row32 = reinterpret_cast<const uint32_t*>(row);
          if (FMT == WT_Q4K) {
            unpack_q4k(row, j, o);
          } else if (FMT == WT_Q5K) {
            unpack_q5k_row(row, j, o);
          } else if (FMT == WT_Q80) {
            if (g) h ? unpack_q80_row<3>(row, o) : unpack_q80_row<1>(row, o);
            else h ? unpack_q80_row<2>(row, o) : unpack_q80_row<0>(row, o);
          } else if (FMT == WT_Q6K) {
            h ? unpack_q6k_half<1>(half, o) : unpack_q6k_half<0>(half, o);
          } else if (dt == INFR_CUDA_DT_Q6K) {
            unpack_q6k(row32, mis * 8, h, g, o);
          } else if (dt == INFR_CUDA_DT_Q8_0) {
            unpack_q80([&](int i) { return row32[17 * j + i]; }, o);
          } else if (dt == INFR_CUDA_DT_Q5K) {
            unpack_k45_words<true>(row32, j, o);
          } else if (dt == INFR_CUDA_DT_Q4K) {
            unpack_k45_words<false>(row32, j, o);
          } else {
            unpack_codes(dt, row + mis, j, o);
          }
          if (h == 1 && FMT != WT_Q6K) {
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars.empty_raw[rp.s]);
          }
          if (TRACED && blk < 4) trace_stamp(tr, 66 + 64 * MODE + 8 * blk + 4 * h);
          if (!wt_wait(&bars.empty_a[ap.s], ap.phase ^ 1)) { ok = false; break; }
          fence_after_sync();
          tmem_st_32x32(a_addr + 64u * ap.s, o);
          fence_before_sync();
          __syncwarp();
          if (lane == 0) arrive_first(&bars.full_a[ap.s]);
          if (TRACED && blk < 4) trace_stamp(tr, 67 + 64 * MODE + 8 * blk + 4 * h);
          if (TRACED && blk < 4 && h == 0) {  // the block's second step has its raw blocks already
            trace_stamp(tr, 68 + 64 * MODE + 8 * blk);
            trace_stamp(tr, 69 + 64 * MODE + 8 * blk);
          }
          ap.next(W_A_STAGES);
          if (FMT != WT_Q6K || h == 1) ap.next(W_A_STAGES);
          if (FMT == WT_Q6K && h == 1) ap.next(W_A_STAGES);
        }
        if (!ok) break;
        rp.next(w.rb);
      }
      if (!ok) break;
      if (!wt_wait(&bars.done, d_phase)) { ok = false; break; }
      d_phase ^= 1;
      fence_after_sync();
      if (TRACED) trace_stamp(tr, 42 + 4 * MODE);
      const float clamp = e < p.n_expert ? p.clamp : 0.f;  // the shared expert's segment is not clamped
      // the down kernel's operand: [K step][rows of the tile][128 B], swizzled like its image in shared memory
      unsigned char* act = reinterpret_cast<unsigned char*>(p.act) + (size_t)row0 * p.nff * 2 + (size_t)(2 * blk0 + (q >> 1)) * rows_valid * 128;
      // warps of one lane quarter share the tile's tokens, 16 at a time
      for (int t0 = 16 * (warp >> 2); t0 < rows_valid; t0 += 64) {
        const uint32_t tq = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)t0;
        float v[2][2][8];  // [accumulator][16 lanes][fragment]
        tmem_ld_16x16_quad(tq, tq + (16u << 16), tq + WN, tq + WN + (16u << 16), v[0][0], v[0][1], v[1][0], v[1][1]);
        if (MODE == 0) {
          if (p.act_kind == INFR_CUDA_ACT_SILU && clamp == 0.f) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              // accumulators are 256 x the products: SiLU(g) u = g u / (1 + 2^(-log2(e) g))
              float& ga = v[0][i >> 3][i & 7];
              const float ex = exp2_approx(ga * (-1.44269504f * W_POSTSCALE));
              ga = __fdividef(ga * W_POSTSCALE, 1.0f + ex) * (v[1][i >> 3][i & 7] * W_POSTSCALE);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              v[0][i >> 3][i & 7] = gated_act_general(p.act_kind, clamp, v[0][i >> 3][i & 7] * W_POSTSCALE, v[1][i >> 3][i & 7] * W_POSTSCALE);
          }
          const int mi = lane >> 3;  // transposed on the way out: a patch row is a token's 32 positions of this lane quarter
#pragma unroll
          for (int h = 0; h < 2; ++h)
            stmatrix_x4_trans(patch_u + ((lane & 7) + 8 * (mi >> 1)) * 80 + (2 * h + (mi & 1)) * 16, f16x2_sat(v[0][h][0], v[0][h][1]),
                              f16x2_sat(v[0][h][2], v[0][h][3]), f16x2_sat(v[0][h][4], v[0][h][5]), f16x2_sat(v[0][h][6], v[0][h][7]));
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int t = (lane >> 2) + 8 * i, c = lane & 3;
            const uint4 x = *reinterpret_cast<const uint4*>(patch + t * 80 + c * 16);
            if (t0 + t < rows_valid) *reinterpret_cast<uint4*>(act + (size_t)(t0 + t) * 128 + (((4 * (q & 1) + c) ^ (t & 7)) << 4)) = x;
          }
          __syncwarp();
        } else {
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            if (m == 1 && lone) break;
            const int mw = lone ? rank : m, f0 = blk0 * WR + (mw * 4 + q) * 32;  // first of the lane quarter's 32 places among the output features
            if (p.y_packed) {
              // the combine kernel is the only reader: this thread's four outputs of a token (8 places apart) as one item
#pragma unroll
              for (int k = 0; k < 4; ++k) {  // tokens 8 (k >> 1) + 2 (lane % 4) + (k & 1)
                const int i0 = 4 * (k >> 1) + (k & 1), t = t0 + 8 * (k >> 1) + 2 * (lane & 3) + (k & 1);
                uint2 hi;
                uint32_t lo;
                pack_y4(v[m][0][i0], v[m][0][i0 + 2], v[m][1][i0], v[m][1][i0 + 2], hi, lo);
                if (t < rows_valid) {
                  unsigned char* row = reinterpret_cast<unsigned char*>(p.y) + (size_t)(row0 + t) * p.ne * 3;
                  reinterpret_cast<uint2*>(row)[f0 / 4 + (lane >> 2)] = hi;
                  reinterpret_cast<uint32_t*>(row + 2 * p.ne)[f0 / 4 + (lane >> 2)] = lo;
                }
              }
            } else if (w.row_shift == 0) {
#pragma unroll
              for (int cg = 0; cg < 2; ++cg) {  // eight tokens at a time
                float* pf = reinterpret_cast<float*>(patch);
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                  for (int i = 0; i < 4; ++i)
                    pf[(2 * (lane & 3) + (i & 1)) * 36 + h * 16 + (i >> 1) * 8 + (lane >> 2)] = v[m][h][4 * cg + i] * W_POSTSCALE;
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                  const int t = (lane >> 3) + 4 * i, c = lane & 7;
                  const float4 x = *reinterpret_cast<const float4*>(pf + t * 36 + c * 4);
                  if (t0 + 8 * cg + t < rows_valid)
                    *reinterpret_cast<float4*>(p.y + (size_t)(row0 + t0 + 8 * cg + t) * p.ne + f0 + c * 4) = x;
                }
                __syncwarp();
              }
            } else {
              // outputs of neighbouring features are in different warps: the four of these tokens put theirs in order together
              // (4-byte stores a whole row_shift apart: 1500 tokens of Q5_K / Q5_K / Q6_K 320 -> 380 us)
              const int sh = w.row_shift, p0 = sh >= 2 ? q : (q >> 1) * 64 + (q & 1), pl = sh >= 2 ? 4 : 2;  // lane l's place: p0 + pl l
              float* pf = reinterpret_cast<float*>(patches + (size_t)(warp & ~3) * W_PATCH);  // [8 tokens][132]
#pragma unroll
              for (int cg = 0; cg < 2; ++cg) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                  for (int i = 0; i < 4; ++i)
                    pf[(2 * (lane & 3) + (i & 1)) * 132 + p0 + pl * (h * 16 + (i >> 1) * 8 + (lane >> 2))] = v[m][h][4 * cg + i] * W_POSTSCALE;
                if (ok) ok = meet(&bars.patch[warp >> 2], m_phase);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                  const int t = q + 4 * i;
                  const float4 x = *reinterpret_cast<const float4*>(pf + t * 132 + lane * 4);
                  if (t0 + 8 * cg + t < rows_valid)
                    *reinterpret_cast<float4*>(p.y + (size_t)(row0 + t0 + 8 * cg + t) * p.ne + blk0 * WR + (sh == 3 ? 8 * lane + 4 * mw : mw * 128 + 4 * lane)) = x;
                }
                if (ok) ok = meet(&bars.patch[warp >> 2], m_phase);
              }
            }
          }
        }
      }
      fence_before_sync();
      __syncwarp();
      if (lane == 0) arrive_first(&bars.drained);
      if (TRACED) trace_stamp(tr, 43 + 4 * MODE);
    }
    if (!ok && lane == 0) atomicExch(&p.status->timeout, 5 + MODE);
  } else if (warp == W_MMA_WARP) {
    // ---- MMA issue: the first CTA's warp waits, one elected lane issues for both; the second's passes on that its tokens are there ----
    RingPos bp, ap;
    if (rank != 0) {
      if (MODE == 0) ok = ok && relay_tokens<PER, B_STAGES>(bars, n_jobs, 4 * kb, 0, RELAYS);
      for (int it = 0; ok && wt_job(it) < n_jobs; ++it)
        for (int step = 0; step < 4 * kb; ++step) {
          bp.next(B_STAGES);
          ap.next(W_A_STAGES);
        }
    } else {
      const uint64_t db0 = smem_desc_k_major_swz128(b_ring, 0);
      uint32_t r_phase = 1;
      for (int it = 0; ok; ++it) {
        const int job = wt_job(it);
        if (job >= n_jobs) break;
        const JobBlock jb = wt_block(job, w.n_pair, w.n_blk, 0);
        const uint32_t idesc = idesc_f16_f32(256, (__shfl_sync(0xFFFFFFFFu, __ldcg(p.tile_rows + jb.tile), 0) + 31) & ~31);
        ok = __all_sync(0xFFFFFFFFu, wt_wait(&bars.drained, r_phase));
        if (!ok) break;
        r_phase ^= 1;
        for (int step = 0; step < 4 * kb; ++step) {
          ok = __all_sync(0xFFFFFFFFu, (MODE == 0 ? pair_wait(&bars.full_b[bp.s], bp.phase) : wt_wait(&bars.full_b[bp.s], bp.phase)) &&
                                          wt_wait(&bars.full_a[ap.s], ap.phase));
          if (!ok) break;
          fence_after_sync();
          if (elect_one()) {
            const uint64_t db = db0 + (uint64_t)(bp.s * (W_B_STAGE >> 4));
            const uint32_t a = W_A_COL + 64u * ap.s, acc = step > 0;
            unsigned long long* tr = TRACED && job == p.trace_tile * w.n_pair && step < 16 ? p.trace : nullptr;
            if (TRACED) trace_write(tr, 96 + 64 * MODE + 2 * step);
            if (MODE == 0) fence_proxy_async();
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              mma_f16_ta(tmem, a + 8 * k, db + 2 * k, idesc, k > 0 ? 1u : acc);
              if (!ODD || !jb.lone) mma_f16_ta(tmem + WN, a + 32 + 8 * k, db + 2 * k, idesc, k > 0 ? 1u : acc);
            }
            commit_pair(&bars.empty_a[ap.s]);
            commit_pair(&bars.empty_b[bp.s]);
            if (step == 4 * kb - 1) commit_pair(&bars.done);
            if (TRACED) trace_write(tr, 97 + 64 * MODE + 2 * step);
          }
          __syncwarp();
          bp.next(B_STAGES);
          ap.next(W_A_STAGES);
        }
      }
    }
    // every commit that this CTA was promised has arrived before either leaves
    for (int i = 0; i < B_STAGES && ok; ++i, bp.next(B_STAGES)) ok = wt_wait(&bars.empty_b[bp.s], bp.phase ^ 1);
    for (int i = 0; i < W_A_STAGES && ok; ++i, ap.next(W_A_STAGES)) ok = wt_wait(&bars.empty_a[ap.s], ap.phase ^ 1);
    if (!ok && lane == 0) atomicExch(&p.status->timeout, 5 + MODE);
  } else if (warp < RAW_WARP) {
    // ---- token operand ----
    RingPos bp;
    if (MODE == 1) {
      // the tile's activations: [K step][rows of the tile][128 B], swizzled - this CTA's half as copies of 16 rows, a lane each
      // (past the tile's last row they read on into the next step: columns of the accumulators that nothing looks at)
      pdl_wait();
      for (int it = 0; ok; ++it) {
        const int job = wt_job(it);
        if (job >= n_jobs) break;
        const int tile = job / w.n_pair, rows_valid = __ldcg(p.tile_rows + tile), half = (rows_valid + 31) >> 5;  // copies of 16 rows
        const int y0 = __ldcg(p.tile_row0 + tile) * (p.nff >> 6) + 16 * (rank * half + lane);
        for (int step = 0; step < 4 * kb; ++step) {
          if (!wt_wait(&bars.empty_b[bp.s], bp.phase ^ 1)) { ok = false; break; }
          if (rank == 0 && lane == 0) mbar_arrive_expect_tx(&bars.full_b[bp.s], (uint32_t)half * 2 * 16 * 128);
          if (lane < half) tma_load_2d_first(b_ring + (size_t)bp.s * W_B_STAGE + lane * 2048, &tm_act, 0, y0 + step * rows_valid, &bars.full_b[bp.s]);
          __syncwarp();
          bp.next(B_STAGES);
        }
      }
    } else {
      // Token rows from where they are: eight lanes per row and K step, 16 bytes each, straight into the swizzled operand
      // image; two warps share a step (four rows out of every eight each), the two pairs alternate.  (Gathering TMA
      // copies, four rows each, took 18 cycles per row: twice the tensor-core time of the step.)
      const int tw = warp - W_TOK_WARP, r8 = (tw & 1) * 4 + (lane >> 3), c = lane & 7;
      const uint32_t dst0 = smem_u32(b_ring) + (uint32_t)r8 * 128u + (uint32_t)((c ^ r8) << 4);
      const uint4* tok = reinterpret_cast<const uint4*>(p.xg) + c;
      const int n_sorted = __ldcg(w.seg_off + w.n_seg_routed);
      if (tw & 2) bp.next(B_STAGES);
      for (int it = 0; ok; ++it) {
        const int job = wt_job(it);
        if (job >= n_jobs) break;
        const int tile = job / w.n_pair;
        const int row0 = __ldcg(p.tile_row0 + tile), rows_valid = __ldcg(p.tile_rows + tile), ni = ((rows_valid + 31) >> 5) * 2;
        uint32_t src[WN / 16];  // rows 8 i + r8 of this CTA's half, in units of 16 bytes
#pragma unroll
        for (int i = 0; i < WN / 16; ++i) {
          if (i < ni) {
            const int pos = row0 + min(8 * (rank * ni + i) + r8, rows_valid - 1);  // past the end: the last row once more
            const int t = w.pair_of_pos == nullptr ? pos : pos < n_sorted ? __ldcg(w.pair_of_pos + pos) / w.n_used : pos - n_sorted;
            src[i] = (uint32_t)t * (uint32_t)(p.ne >> 3);
          }
        }
        for (int step = tw >> 1; step < 4 * kb; step += 2) {
          if (!wt_wait(&bars.empty_b[bp.s], bp.phase ^ 1)) { ok = false; break; }
          const uint32_t dst = dst0 + (uint32_t)bp.s * W_B_STAGE;
          const uint4* ts = tok + step * 8;
#pragma unroll
          for (int i = 0; i < WN / 16; ++i)
            if (i < ni) cp_async16(dst + i * 1024, ts + src[i]);
          cp_async_arrive(&bars.full_b[bp.s]);
          bp.next(B_STAGES);
          bp.next(B_STAGES);
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
    if (!ok && lane == 0) atomicExch(&p.status->timeout, 5 + MODE);
  } else if (RELAYS > 1 && warp > RAW_WARP) {
    if (rank != 0 && ok && !relay_tokens<PER, B_STAGES>(bars, n_jobs, 4 * kb, warp - RAW_WARP, RELAYS) && lane == 0) atomicExch(&p.status->timeout, 5 + MODE);
  } else if (warp < RAW_WARP + RAW_WARPS) {
    // ---- raw blocks ----
    RingPos rp;
    for (int it = 0; ok; ++it) {
      const int job = wt_job(it);
      if (job >= n_jobs) break;
      const JobBlock jb = wt_block(job, w.n_pair, w.n_blk, rank);
      const int blk0 = jb.blk0, e = __ldcg(p.tile_expert + jb.tile);
      const bool shared_seg = e >= p.n_expert;
      if (wt_tiled(FMT)) {
        if (warp != RAW_WARP || lane != 0) break;  // one thread issues the tiled copies
        // rows of one expert in the bank: nff, or 2 nff where gate and up share a bank (the up map then starts nff rows in)
        const int r0 = MODE == 0 ? (shared_seg ? 0 : e * p.gu_rows) + blk0 * 128 : (shared_seg ? 0 : e * p.ne) + blk0 * WR;
        for (int blk = 0; blk < kb; ++blk) {
          if (!wt_wait(&bars.empty_raw[rp.s], rp.phase ^ 1)) { ok = false; break; }
          unsigned char* dst = raw_ring + (size_t)rp.s * w.raw_stage;
          if (FMT == WT_Q6K) {
            const int n = 1 << w.row_shift, i0 = ODD && jb.lone && n == 8 ? 4 * rank : 0, i1 = ODD && jb.lone && n == 8 ? i0 + 4 : n;
            // the rows of one place among 2^row_shift rows per copy, from the 16-byte boundary at or ahead of the block (a box that
            // runs on past the last block's row is filled up with zeros)
            mbar_arrive_expect_tx(&bars.full_raw[rp.s], (w.raw_stage >> w.row_shift) * (i1 - i0));
            for (int i = i0; i < i1; ++i)
              tma_load_2d(dst + i * (w.raw_stage >> w.row_shift), shared_seg ? &tm_s0 : &tm_w0, (((int)Q6K_BLOCK_BYTES * (i * kb + blk)) & ~15) >> 1,
                          r0 >> w.row_shift, &bars.full_raw[rp.s]);
            rp.next(w.rb);
            continue;
          }
          const int x = blk * (int)(w.raw_pitch >> 1);  // in half-words
          const bool lone = ODD && jb.lone;
          mbar_arrive_expect_tx(&bars.full_raw[rp.s], lone ? w.raw_stage / 2 : w.raw_stage);
          if (!lone || rank == 0) tma_load_2d(dst, shared_seg ? &tm_s0 : &tm_w0, x, r0, &bars.full_raw[rp.s]);
          if (!lone || rank != 0)
            tma_load_2d(dst + 128 * w.raw_pitch, shared_seg ? &tm_s1 : &tm_w1, x, r0 + (MODE == 0 ? 0 : 128), &bars.full_raw[rp.s]);
          rp.next(w.rb);
        }
      } else {
        // Whole words over a block's bytes: a block off a word boundary takes the half-word ahead of it, one that ends off
        // a word boundary the half-word behind it (inside the bank: its block count is even).  One instruction per row and
        // 32 words; the words left over of as many rows as fit share one.
        const int lw = warp - RAW_WARP;
        for (int blk = 0; blk < kb; ++blk) {
          if (!wt_wait(&bars.empty_raw[rp.s], rp.phase ^ 1)) { ok = false; break; }
#pragma unroll
          for (int half = 0; half < 2; ++half) {  // gate and up rows, or the two halves of the output features
            const int dt = MODE == 1 ? p.down_dt : half ? p.up_dt : p.gate_dt;
            const uint8_t* bank = MODE == 1 ? (shared_seg ? p.sh_down : p.down + (size_t)e * p.down_stride)
                                            : half ? (shared_seg ? p.sh_up : p.up + (size_t)e * p.up_stride)
                                                   : (shared_seg ? p.sh_gate : p.gate + (size_t)e * p.gate_stride);
            const uint32_t chunk = (uint32_t)row_bytes(dt, 256);
            const uint32_t words = (chunk + 2) >> 2, full = words >> 5, tail = words & 31u, tail_rows = tail ? 32u / tail : 1u;
            const size_t pitch = (size_t)chunk * kb;
            const uint32_t dst0 = smem_u32(raw_ring) + rp.s * w.raw_stage + (uint32_t)half * 128u * w.raw_pitch;
            const uintptr_t src = reinterpret_cast<uintptr_t>(bank + (size_t)(MODE == 0 ? blk0 * 128 : blk0 * WR + half * 128) * pitch + (size_t)blk * chunk);
            if (full) {
              uintptr_t a = src + lw * pitch + 4 * lane;
              uint32_t d = dst0 + lw * w.raw_pitch + 4 * lane;
#pragma unroll 4
              for (int r = lw; r < 128; r += RAW_WARPS, a += RAW_WARPS * pitch, d += RAW_WARPS * w.raw_pitch) {
                cp_async4(d, reinterpret_cast<const void*>(a & ~(uintptr_t)3));
                if (full > 1) cp_async4(d + 128, reinterpret_cast<const void*>((a & ~(uintptr_t)3) + 128));
              }
            }
            if (tail) {
              const uint32_t t_row = lane / tail + lw * tail_rows, t_word = 32u * full + lane % tail, stride = RAW_WARPS * tail_rows;
              const bool on = lane < tail_rows * tail;
              uintptr_t a = src + t_row * pitch + 4 * t_word;
              uint32_t d = dst0 + t_row * w.raw_pitch + 4 * t_word;
#pragma unroll 4
              for (uint32_t r = t_row; r < 128 + stride; r += stride, a += stride * pitch, d += stride * w.raw_pitch)
                if (on && r < 128) cp_async4(d, reinterpret_cast<const void*>(a & ~(uintptr_t)3));
            }
          }
          cp_async_arrive(&bars.full_raw[rp.s]);
          rp.next(w.rb);
        }
      }
    }
    if (!wt_tiled(FMT)) asm volatile("cp.async.wait_all;" ::: "memory");
    if (!ok && lane == 0) atomicExch(&p.status->timeout, 5 + MODE);
  }
  fence_before_sync();
  __syncwarp();
  pair_sync();
  __syncwarp();
  if (warp == W_MMA_WARP) tmem_dealloc_pair(s_tmem);
}

// A bank as a 2-D tensor of half-words [rows][row bytes / 2]; box: 256 weights (`chunk` bytes) of `box_rows` rows.
bool raw_rows_map(CUtensorMap* tm, const uint8_t* base, size_t rows, size_t row_bytes, uint32_t chunk, uint32_t box_rows = 128) {
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)row_bytes / 2, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)row_bytes};
  const cuuint32_t box[2] = {chunk / 2, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return enc(tm, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<uint8_t*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int wt_format(int dt0, int dt1, bool down) {
  if (dt0 == dt1) {
    if (dt0 == INFR_CUDA_DT_Q4K) return WT_Q4K;
    if (dt0 == INFR_CUDA_DT_Q5K) return WT_Q5K;
    if (dt0 == INFR_CUDA_DT_Q8_0) return WT_Q80;
    if (dt0 == INFR_CUDA_DT_Q6K && down) return WT_Q6K;
  }
  return WT_ANY;
}

// Bytes of 256 weights of a row in the raw stage.
uint32_t raw_pitch_of(int fmt, int dt) {
  if (fmt == WT_Q6K) return W_Q6K_BOX;
  if (wt_tiled(fmt)) return (uint32_t)row_bytes(dt, 256);  // 36, 44 or 68 words: 16-byte pieces of eight rows in different banks
  const uint32_t words = ((uint32_t)row_bytes(dt, 256) + 2 + 3) / 4;  // room for the half-word ahead
  return (words | 1) * 4;
}

template <int MODE, int FMT>
int32_t launch_wt(infr_cuda_ctx* ctx, WtParams w, const CUtensorMap (&tm)[5], int max_tiles) {
  // the token stages, and as many raw stages as fit beside them, two at least
  const size_t patches = (size_t)(W_PRODUCERS / 32) * W_PATCH;
  constexpr uint32_t b_ring = wt_b_stages(MODE, FMT) * W_B_STAGE;
  const size_t room = 227 * 1024 - 1024 - 1024 - patches - b_ring;  // alignment slack, static shared memory
  w.rb = (int)std::min<size_t>(W_MAX_RAW, room / w.raw_stage);
  if (w.rb < 2) return fail(ctx, INFR_CUDA_ERR_UNSUPPORTED, "grouped GEMM: blocks too large for the raw ring");
  const size_t smem = 1024 + b_ring + (size_t)w.rb * w.raw_stage + patches;
  constexpr bool MAY_BE_ODD = MODE == 1;  // gate/up: blocks of 128 features, of 256 k
  const bool odd = w.n_blk & 1;
  auto kern = w.g.trace != nullptr ? (odd ? k_wt_gemm<MODE, FMT, true, MAY_BE_ODD> : k_wt_gemm<MODE, FMT, true, false>)
                                   : (odd ? k_wt_gemm<MODE, FMT, false, MAY_BE_ODD> : k_wt_gemm<MODE, FMT, false, false>);
  cudaError_t e = ensure_smem(reinterpret_cast<const void*>(kern), smem);
  if (e != cudaSuccess) return check_cuda(ctx, e, "grouped GEMM: shared-memory attribute");
  const long long jobs = (long long)max_tiles * w.n_pair;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (unsigned)std::min<long long>(jobs, ctx->sm_count / 2));
  cfg.blockDim = dim3(W_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim = {2, 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  e = cudaLaunchKernelEx(&cfg, kern, w, tm[0], tm[1], tm[2], tm[3], tm[4]);
  if (e != cudaSuccess) return check_cuda(ctx, e, "grouped GEMM launch");
  ctx->launches += 1;
  return check_cuda(ctx, cudaGetLastError(), "grouped GEMM launch");
}

}  // namespace

int wt_tile_rows() { return WN; }

// A Q6_K row of 256 k weights is 210 k bytes: 1, 2, 4 or 8 rows are whole 16-byte pieces.
int wt_y_shift(int down_dt, int nff) {
  if (wt_format(down_dt, down_dt, true) != WT_Q6K) return 0;
  int sh = 0;
  while ((row_bytes(down_dt, nff) << sh) % 16) ++sh;
  return sh;
}

int32_t launch_wt_grouped(infr_cuda_ctx* ctx, const GroupedParams& p, const WtTokens& t, int max_tiles) {
  WtParams w = {};
  w.g = p;
  w.pair_of_pos = t.pair_of_pos;
  w.seg_off = t.seg_off;
  w.n_seg_routed = t.n_seg_routed;
  w.n_used = t.n_used;
  CUtensorMap tm[5] = {};
  bool ok = true;

  // gate / up.  A bank's rows are one 2-D tensor; with gate and up in one bank an expert has 2 nff rows and the up map
  // starts nff rows in (and ends with the bank)
  w.n_blk = p.nff / 128;
  w.n_pair = (w.n_blk + 1) / 2;
  w.k_blocks = p.ne / 256;
  int fmt = wt_format(p.gate_dt, p.up_dt, false);
  w.raw_pitch = std::max(raw_pitch_of(fmt, p.gate_dt), raw_pitch_of(fmt, p.up_dt));
  w.raw_stage = WR * w.raw_pitch;
  if (wt_tiled(fmt)) {
    const size_t rb = row_bytes(p.gate_dt, p.ne), bank_rows = (size_t)p.n_expert * p.gu_rows;
    ok = raw_rows_map(&tm[0], p.gate, bank_rows, rb, w.raw_pitch) && raw_rows_map(&tm[1], p.up, bank_rows - ((size_t)p.gu_rows - p.nff), rb, w.raw_pitch);
    if (ok && p.sh_gate) ok = raw_rows_map(&tm[2], p.sh_gate, p.nff, rb, w.raw_pitch) && raw_rows_map(&tm[3], p.sh_up, p.nff, rb, w.raw_pitch);
    if (!ok) return fail(ctx, INFR_CUDA_ERR_CUDA, "grouped GEMM: the driver refused a tensor map for the expert banks");
  }
  int32_t rc = fmt == WT_Q4K   ? launch_wt<0, WT_Q4K>(ctx, w, tm, max_tiles)
               : fmt == WT_Q5K ? launch_wt<0, WT_Q5K>(ctx, w, tm, max_tiles)
               : fmt == WT_Q80 ? launch_wt<0, WT_Q80>(ctx, w, tm, max_tiles)
                               : launch_wt<0, WT_ANY>(ctx, w, tm, max_tiles);
  if (rc) return rc;

  // down
  w.n_blk = p.ne / WR;
  w.n_pair = (w.n_blk + 1) / 2;
  w.k_blocks = p.nff / 256;
  fmt = wt_format(p.down_dt, p.down_dt, true);
  w.raw_pitch = raw_pitch_of(fmt, p.down_dt);
  w.raw_stage = WR * w.raw_pitch;
  w.row_shift = p.y_shift;
  // the activations as a tensor of 128-byte rows: 16 of them a copy
  if (!raw_rows_map(&tm[4], reinterpret_cast<const uint8_t*>(p.act), ((size_t)t.rows_bound + 256) * (p.nff / 64), 128, 128, 16))
    return fail(ctx, INFR_CUDA_ERR_CUDA, "grouped GEMM: the driver refused a tensor map for the activations");
  if (wt_tiled(fmt)) {
    const size_t rb = row_bytes(p.down_dt, p.nff) << w.row_shift;
    const uint32_t box_rows = fmt == WT_Q6K ? (uint32_t)WR >> w.row_shift : 128u;
    ok = raw_rows_map(&tm[0], p.down, (size_t)p.n_expert * p.ne >> w.row_shift, rb, w.raw_pitch, box_rows);
    if (ok && p.sh_down) ok = raw_rows_map(&tm[2], p.sh_down, (size_t)p.ne >> w.row_shift, rb, w.raw_pitch, box_rows);
    tm[1] = tm[0];
    tm[3] = tm[2];
    if (!ok) return fail(ctx, INFR_CUDA_ERR_CUDA, "grouped GEMM: the driver refused a tensor map for the down bank");
  }
  return fmt == WT_Q4K   ? launch_wt<1, WT_Q4K>(ctx, w, tm, max_tiles)
         : fmt == WT_Q5K ? launch_wt<1, WT_Q5K>(ctx, w, tm, max_tiles)
         : fmt == WT_Q80 ? launch_wt<1, WT_Q80>(ctx, w, tm, max_tiles)
         : fmt == WT_Q6K ? launch_wt<1, WT_Q6K>(ctx, w, tm, max_tiles)
                         : launch_wt<1, WT_ANY>(ctx, w, tm, max_tiles);
}

cudaError_t publish_codebooks_tmem(const unsigned char* const* tables) { return publish_codebooks(tables); }

}  // namespace infr

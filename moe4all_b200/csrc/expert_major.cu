// Small-m expert FFN, expert-major: one CTA owns one expert (and a tile of its rows) for ALL tokens of
// the call that were routed to it.
//
//   k_em_bucket  : (token, rank) pairs grouped by expert into segments of at most 8 pairs; integer sums
//                  of the fixed-point activations per 32-element sub-block
//   k_em_gateup  : act[pair, f] = act_fn(W_gate[e][f,:]·x_tok) * (W_up[e][f,:]·x_tok)       (Q4_K banks)
//   k_em_down    : y[pair, i]   = W_down[e][i,:]·act[pair,:]                                 (Q6_K bank)
//   k_em_combine : dst[r, :]    = sum over ranks (rank order) w * y[pair] + shared expert (+ residual)
//
// Reference: the same CPU stages as the per-pair kernels (crates/infr-cpu/src/lib.rs:3873-3907 bucket by
// expert, :4051-4266 expert mat-vecs, :4287-4303 rank-ordered sum).  The reference's GPU backend switches
// from one dispatch per (token, expert) pair to row tiles over an expert's tokens between 8 and 16
// rows (crates/infr-vulkan/src/adapter.rs:253-287) with 32-row tiles for lightly loaded experts
// (crates/infr-vulkan/src/recorder.rs:283, 15219-15225); this file is that middle regime.
//
// Arithmetic: weights stay the GGUF integer codes, activations are 16-bit fixed point in two signed
// 8-bit limbs (X = 256 hi + lo, as in the per-pair kernels), and the products run on the tensor cores'
// integer path: `mma.sync m16n8k32 u8 x s8 -> s32` per 32-element Q4_K sub-block (m16n8k16 per 16-element
// Q6_K scale group), one MMA per limb.  The integer sums are exact; the 6-bit (8-bit) block scales are
// applied to them in integers as well and a block's total is converted to f32 once.  A weight word is
// fetched and masked once per CTA and multiplied against up to 8 token rows, so the cost per weight does
// not grow with the tokens an expert sees, and the kernels stream the distinct experts' bytes once
// (1-D bulk async copies into shared memory, never multicast).
#include "kernels.cuh"
#include "tma.cuh"

namespace infr {

namespace {

constexpr int EM_FEAT = 32;         // gate/up: features per CTA
constexpr int EM_MAX_STAGES = 4;
constexpr int EM_SEG = 8;           // token rows per segment = the N extent of one MMA
constexpr int EM_NARROW = 4;        // segments of up to this many: both limbs of a token as columns of one MMA

__device__ __forceinline__ void mma_u8s8_k32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mma_u8s8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
               : "r"(a0), "r"(a1), "r"(b0));
}

// The part of a block's result that the offsets of its codes make, sum over the scale groups of (min or scale) x (sum of the
// group's fixed-point elements), is a small contraction of its own.  The sums, below 2^20, are split into three bytes, the upper one
// signed, and take one MMA of K 16 each: in integers, exact.  (As multiply-adds of every thread, with the sums and the mins fetched and
// taken apart per group, they were a fifth of the instructions, which are what these kernels are bound by.  Gate/up and down, us with the
// wait for the router: 32 rows of 256 experts of 512 67 / 53 -> 65 / 46, 64 rows of 28 MB experts 607 / 580 -> 558 / 554.)
#define EM_OFFSET_MMA(NAME, A, B)                                                                                          \
  __device__ __forceinline__ void NAME(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {                               \
    c[0] = c[1] = c[2] = c[3] = 0;                                                                                         \
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32." A "." B ".s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"      \
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(b0));                            \
  }
EM_OFFSET_MMA(mma_u8u8, "u8", "u8")
EM_OFFSET_MMA(mma_u8s8, "u8", "s8")
EM_OFFSET_MMA(mma_s8u8, "s8", "u8")
EM_OFFSET_MMA(mma_s8s8, "s8", "s8")
#undef EM_OFFSET_MMA

// Rows g and g + 8 (a0, a1; SGN: signed bytes) against the sums of the tokens of this thread's accumulator columns, added to mv[row][token].
// b0, b1, b2: the bytes of the sums of column g's token; NARROW: b0 is byte g & 1 of token g / 2's, b1 is not used.
template <bool NARROW, bool SGN, int NT>
__device__ __forceinline__ void offset_sums(uint32_t a0, uint32_t a1, uint32_t b0, uint32_t b1, uint32_t b2, int (&mv0)[NT], int (&mv1)[NT]) {
  int lo[4], mid[4], hi[4];
  SGN ? mma_s8u8(lo, a0, a1, b0) : mma_u8u8(lo, a0, a1, b0);
  if (!NARROW) SGN ? mma_s8u8(mid, a0, a1, b1) : mma_u8u8(mid, a0, a1, b1);
  SGN ? mma_s8s8(hi, a0, a1, b2) : mma_u8s8(hi, a0, a1, b2);
#pragma unroll
  for (int k = 0; k < NT; ++k) {
    mv0[k] = lo[k] + (NARROW ? lo[1] : mid[k]) * 256 + hi[k] * 65536;
    mv1[k] = lo[2 + k] + (NARROW ? lo[3] : mid[2 + k]) * 256 + hi[2 + k] * 65536;
  }
}

// The eight scales, or mins, of a Q4_K block from its header, four to a word (s0, s1, s2: header words 1 to 3).
__device__ __forceinline__ void q4k_scales(uint32_t s0, uint32_t s2, uint32_t (&sc)[2]) {
  sc[0] = s0 & 0x3F3F3F3Fu;
  sc[1] = (s2 & 0x0F0F0F0Fu) | ((s0 >> 2) & 0x30303030u);
}
__device__ __forceinline__ uint32_t q4k_mins(uint32_t s1, uint32_t s2, int upper) {
  return upper ? ((s2 >> 4) & 0x0F0F0F0Fu) | ((s1 >> 2) & 0x30303030u) : s1 & 0x3F3F3F3Fu;
}
__device__ __forceinline__ int byte_of(uint32_t w, int i) { return (int)__byte_perm(w, 0, 0x4440 | i); }

// ---------------------------------------------------------------------------------------------
// bucket: pairs by expert, in segments of at most `seg_cap` pairs; the shared expert's rows are
// appended as segments of "expert" n_expert over pair ids P + r.  One CTA.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) k_em_bucket(EmParams p, int seg_cap) {
  __shared__ int s_cnt[1024], s_off[1024];
  __shared__ int s_wc[32], s_wsg[32], s_ws[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, E = p.n_expert, P = p.rows * p.n_used;
  pdl_trigger();
  // Two passes over the same code: the first, while the router still runs, without pairs and without stores, has the second find
  // its instructions cached.  A thread keeps its pairs' experts and their ranks inside them (the count before its own) in
  // registers (32 rows, top-8 of 256: 3.2 - 5.5 -> 2.8 us behind the router).  With these the kernel has 58 registers and fits beside no
  // CTA of the router; held to 32, which does, it made the layer 0 - 3 us slower from 33 to 64 rows (40 rows 124.9 -> 128.1).
  constexpr int KEEP = 3;  // covers eleven pairs per expert of 256; more are read again
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    const bool live = pass != 0;
    const int n_pairs = live ? P : 0;
    s_cnt[tid] = 0;
    if (live) {
      pdl_wait();
      // sums of the fixed-point activations per 32-element sub-block (the Q4_K `min` term needs them).
      // xq_* come from the kernel before this one in the stream.
      if (!p.xsum_ready) {  // (a call that only runs the expert stages: no kernel of its own made the fixed-point copy)
        const int nsb = p.ne / 32, total = p.rows * nsb;
        for (int i = tid; i < total; i += 1024) {
          const int r = i / nsb, sb = i - r * nsb;
          const int4* lo = reinterpret_cast<const int4*>(p.xq_lo + (size_t)r * p.ne + sb * 32);
          const int4* hi = reinterpret_cast<const int4*>(p.xq_hi + (size_t)r * p.ne + sb * 32);
          int l = 0, h = 0;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int4 a = __ldcg(lo + q), b = __ldcg(hi + q);
            l = __dp4a(0x01010101, a.x, l); l = __dp4a(0x01010101, a.y, l); l = __dp4a(0x01010101, a.z, l); l = __dp4a(0x01010101, a.w, l);
            h = __dp4a(0x01010101, b.x, h); h = __dp4a(0x01010101, b.y, h); h = __dp4a(0x01010101, b.z, h); h = __dp4a(0x01010101, b.w, h);
          }
          p.xsum[i] = h * 256 + l;
        }
      }
    }
    auto expert_of = [&](int pair) {
      int e = __ldcg(p.ids + pair);
      if (e < 0) return -1;  // a pair another rank serves
      if (e >= E) {
        p.status->bad_index = 1;
        e = E - 1;
      }
      if (p.ep_n != 0 && ((uint32_t)e < p.ep_lo || (uint32_t)e >= p.ep_lo + p.ep_n)) return -1;
      return e;
    };
    int my_e[KEEP], my_rank[KEEP];
#pragma unroll
    for (int u = 0; u < KEEP; ++u) my_e[u] = tid + u * 1024 < n_pairs ? expert_of(tid + u * 1024) : -1;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < KEEP; ++u) my_rank[u] = my_e[u] >= 0 ? atomicAdd(&s_cnt[my_e[u]], 1) : 0;
    if (n_pairs > KEEP * 1024) {
      __syncthreads();  // the kept pairs rank first
      for (int i = tid + KEEP * 1024; i < n_pairs; i += 1024) {
        const int e = expert_of(i);
        if (e >= 0) atomicAdd(&s_cnt[e], 1);
      }
    }
    __syncthreads();
    // exclusive scans over experts of (pairs, segments): thread e holds expert e
    const int c = tid < E ? s_cnt[tid] : 0, sg = (c + seg_cap - 1) / seg_cap;
    int ic = c, is = sg;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int uc = __shfl_up_sync(0xFFFFFFFFu, ic, o), us = __shfl_up_sync(0xFFFFFFFFu, is, o);
      if (lane >= o) { ic += uc; is += us; }
    }
    if (lane == 31) { s_wc[warp] = ic; s_wsg[warp] = is; }
    __syncthreads();
    if (warp == 0) {
      int wc = s_wc[lane], wsg = s_wsg[lane];
      const int oc = wc, os = wsg;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int uc = __shfl_up_sync(0xFFFFFFFFu, wc, o), us = __shfl_up_sync(0xFFFFFFFFu, wsg, o);
        if (lane >= o) { wc += uc; wsg += us; }
      }
      s_wc[lane] = wc - oc;
      s_wsg[lane] = wsg - os;
      if (lane == 31) { s_ws[0] = wc; s_ws[1] = wsg; }
    }
    __syncthreads();
    const int off = ic - c + s_wc[warp];
    s_off[tid] = off;
    const int n_routed_pairs = s_ws[0], n_routed_seg = s_ws[1];
    // segment table of the routed experts
    for (int k = 0, sgi = is - sg + s_wsg[warp]; k < c; k += seg_cap, ++sgi) {
      p.seg_expert[sgi] = tid;
      p.seg_off[sgi] = off + k;
      p.seg_cnt[sgi] = min(seg_cap, c - k);
    }
    // the shared expert: every row, in row order
    const int n_sh_seg = p.sh_ff ? (p.rows + seg_cap - 1) / seg_cap : 0;
    for (int i = tid; live && i < n_sh_seg; i += 1024) {
      p.seg_expert[n_routed_seg + i] = E;
      p.seg_off[n_routed_seg + i] = n_routed_pairs + i * seg_cap;
      p.seg_cnt[n_routed_seg + i] = min(seg_cap, p.rows - i * seg_cap);
    }
    if (p.sh_ff)
      for (int r = tid; live && r < p.rows; r += 1024) p.seg_pairs[n_routed_pairs + r] = P + r;
    if (live && tid == 0) *p.n_seg = n_routed_seg + n_sh_seg;
    __syncthreads();
    // scatter (the order inside an expert is arrival order; every pair's result is independent of it)
#pragma unroll
    for (int u = 0; u < KEEP; ++u)
      if (my_e[u] >= 0) p.seg_pairs[s_off[my_e[u]] + my_rank[u]] = tid + u * 1024;
    if (n_pairs > KEEP * 1024) {
      // the rest come behind the kept ones of their expert, counted down from its total
      for (int i = tid + KEEP * 1024; i < n_pairs; i += 1024) {
        const int e = expert_of(i);
        if (e >= 0) p.seg_pairs[s_off[e] + atomicSub(&s_cnt[e], 1) - 1] = i;
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// gate/up + activation
// ---------------------------------------------------------------------------------------------
// One 256-weight block of a warp's rows (gate g, gate g + 8, up g, up g + 8 of its feature group: `w`, eight rows on, `box`
// bytes on) against the segment's tokens, added to fg, fu.
//   wide: the 8 MMA columns are 8 tokens, one MMA per limb (x, x + xh); a thread ends with rows g, g + 8 of tokens 2t, 2t + 1.
//   NARROW (at most four tokens, which is most segments of a decode batch): the columns are the two limbs of four
//   tokens side by side, so a sub-block takes one MMA per role and a thread ends with the low and high sums of rows g,
//   g + 8 of token t: half the MMAs, fragment loads and scale multiplies.
template <bool NARROW>
__device__ __forceinline__ void gateup_block(const unsigned char* w, uint32_t box, const unsigned char* x, uint32_t xh, const int* sums, int b,
                                             float (&fg)[4], float (&fu)[4]) {
  constexpr int NT = NARROW ? 1 : 2;  // tokens of a thread
  const int t = threadIdx.x & 3;
  const unsigned char* rows4[4] = {w, w + 8 * Q4K_BLOCK_BYTES, w + box, w + box + 8 * Q4K_BLOCK_BYTES};
  uint4 hdr[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) hdr[r] = *reinterpret_cast<const uint4*>(rows4[r]);
  int svl[4][NT], svh[4][NT], mv[4][NT];  // [row][token]
  uint32_t scales[4][2];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    q4k_scales(hdr[r].y, hdr[r].w, scales[r]);
#pragma unroll
    for (int k = 0; k < NT; ++k) svl[r][k] = svh[r][k] = 0;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t wA[4], wB[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const unsigned char* q = rows4[r] + 16 + 32 * j + 4 * t;
      wA[r] = *reinterpret_cast<const uint32_t*>(q);
      wB[r] = *reinterpret_cast<const uint32_t*>(q + 16);
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int lsb = b * 8 + 2 * j + half;  // sub-block index inside the stage
      const uint32_t b0 = *reinterpret_cast<const uint32_t*>(x + lsb * 32), b1 = *reinterpret_cast<const uint32_t*>(x + lsb * 32 + 16);
      uint32_t a[4][2];
      int sc[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        a[r][0] = (wA[r] >> (4 * half)) & 0x0F0F0F0Fu;
        a[r][1] = (wB[r] >> (4 * half)) & 0x0F0F0F0Fu;
        sc[r] = byte_of(scales[r][j >> 1], 2 * (j & 1) + half);
      }
      int c0[4] = {0, 0, 0, 0}, c1[4] = {0, 0, 0, 0};
      mma_u8s8_k32(c0, a[0][0], a[1][0], a[0][1], a[1][1], b0, b1);
      mma_u8s8_k32(c1, a[2][0], a[3][0], a[2][1], a[3][1], b0, b1);
      if (NARROW) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          svl[r][0] += sc[r] * (r < 2 ? c0[2 * (r & 1)] : c1[2 * (r & 1)]);
          svh[r][0] += sc[r] * (r < 2 ? c0[2 * (r & 1) + 1] : c1[2 * (r & 1) + 1]);
        }
      } else {
        const uint32_t b0h = *reinterpret_cast<const uint32_t*>(x + xh + lsb * 32), b1h = *reinterpret_cast<const uint32_t*>(x + xh + lsb * 32 + 16);
        int h0[4] = {0, 0, 0, 0}, h1[4] = {0, 0, 0, 0};
        mma_u8s8_k32(h0, a[0][0], a[1][0], a[0][1], a[1][1], b0h, b1h);
        mma_u8s8_k32(h1, a[2][0], a[3][0], a[2][1], a[3][1], b0h, b1h);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int k = 0; k < NT; ++k) {
            const int i = 2 * (r & 1) + k;
            svl[r][k] += sc[r] * (r < 2 ? c0[i] : c1[i]);
            svh[r][k] += sc[r] * (r < 2 ? h0[i] : h1[i]);
          }
      }
    }
  }
  {
    // K positions 4 t .. 4 t + 3 are sub-blocks; eight of the sixteen are padding, with no min
    uint32_t mins[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) mins[r] = t < 2 ? q4k_mins(hdr[r].z, hdr[r].w, t) : 0u;
    const int4 sx = *reinterpret_cast<const int4*>(sums + b * 8 + 4 * (t & 1));
    const uint32_t p01 = __byte_perm(sx.x, sx.y, 0x5140), p23 = __byte_perm(sx.z, sx.w, 0x5140);
    const uint32_t b2 = __byte_perm(__byte_perm(sx.x, sx.y, 0x0062), __byte_perm(sx.z, sx.w, 0x0062), 0x5410);
    const uint32_t b0 = __byte_perm(p01, p23, NARROW && (threadIdx.x & 4) ? 0x7632 : 0x5410), b1 = NARROW ? 0u : __byte_perm(p01, p23, 0x7632);
    offset_sums<NARROW, false>(mins[0], mins[1], b0, b1, b2, mv[0], mv[1]);
    offset_sums<NARROW, false>(mins[2], mins[3], b0, b1, b2, mv[2], mv[3]);
  }
  // once per block: value = d * sum(sc * sum(q X)) - dmin * sum(m * sum(X)), X = 256 hi + lo
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const float d = f16_bits_to_f32(hdr[r].x), dm = f16_bits_to_f32(hdr[r].x >> 16);
#pragma unroll
    for (int k = 0; k < NT; ++k) {
      const float v = d * fmaf(256.f, (float)svh[r][k], (float)svl[r][k]) - dm * (float)mv[r][k];
      (r < 2 ? fg : fu)[2 * (r & 1) + k] += v;
    }
  }
}

// Job = (segment of up to 8 token rows, tile of EM_FEAT features, both roles); the CTAs are persistent
// and take jobs blockIdx.x, blockIdx.x + gridDim.x, ...  2 KS consumer warps: warp (fw, ks) owns features
// 16 fw .. 16 fw + 15 and every KS-th block of the row; MMA rows are the 16 gate rows
// and, in a second accumulator set, the 16 up rows, so a thread ends with gate and up of the same
// (feature, token).  The last warp is the producer: per stage it streams KB blocks of every weight row
// (one tiled TMA copy per block and role: a box of 32 rows x 144 bytes out of rows a whole row apart), the
// same K range of the tokens' fixed-point limbs and their sub-block sums (1-D bulk copies), through a
// ring of S stages that runs on across jobs, so the next job's weights arrive while this one is
// computed.  Row pitches are 4 (mod 8) words, which makes every fragment load (eight rows x four
// consecutive words) conflict-free.
// Scales are applied in integers: per block a thread accumulates sc * (limb sums) and m * sum(X) in int32
// (bounded: 8 sub-blocks x 63 x 32 x 15 x 128 < 2^31) and converts once per block.
// What the consumers need of a job, put beside its first stage by the producer, which looks it up a job ahead (the lookups
// are a chain of three L2 reads; made by every warp at both ends of a job they cost as much as a third of it).
struct EmJob {
  int job, e, cnt;  // job < 0: no more
  int pair[8];
  float xs[8], wp[8];  // value of one step of the token's fixed-point row; weight on the expert's input
};

template <int KS>
__global__ void __launch_bounds__((2 * KS + 1) * 32, 2) k_em_gateup(EmParams p, int KB, int S, int xpitch, int gu_rows,
                                                                    const __grid_constant__ CUtensorMap tm_gate,
                                                                    const __grid_constant__ CUtensorMap tm_up,
                                                                    const __grid_constant__ CUtensorMap tm_sh_gate,
                                                                    const __grid_constant__ CUtensorMap tm_sh_up) {
  constexpr int EM_GU_WARPS = 2 * KS;  // consumer warps
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t s_full[EM_MAX_STAGES], s_empty[EM_MAX_STAGES];
  __shared__ float s_red[2][2][32][8];  // [slot][feature group][lane][gate 4 | up 4]
  __shared__ EmJob s_job[2];            // two suffice: the ring holds no more stages than a job has
  __shared__ int s_abort;               // a consumer warp's bounded wait ran out: all consumers leave together

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int nffmax = p.nffmax, tiles_max = nffmax / EM_FEAT;
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&s_empty[s], EM_GU_WARPS);
    }
    mbar_fence_init();
    s_abort = 0;
  }
  __syncthreads();
  pdl_wait();  // the segment table comes from the bucket kernel
  pdl_trigger();
  const int n_jobs = __ldcg(p.n_seg) * tiles_max;
  const int P = p.rows * p.n_used;
  const int n_kc = (p.ne / 256) / KB, nsb = p.ne / 32;
  const int spitch = KB * 8 + 4;  // ints per token of the sub-block sums: a block's are on a 16-byte boundary
  // stage layout: weights [KB blocks][2 roles][EM_FEAT rows][144] | x limbs [2][8 tokens][xpitch] | sub-block sums [8][spitch] ints
  constexpr uint32_t BOX = EM_FEAT * Q4K_BLOCK_BYTES;  // one block of one role's rows
  const uint32_t w_bytes = (uint32_t)KB * 2 * BOX, x_bytes = (uint32_t)16 * xpitch, s_bytes = (uint32_t)8 * spitch * 4;
  const uint32_t stage_bytes = w_bytes + x_bytes + s_bytes;
  uint32_t it = 0;  // stages used so far by this CTA (both roles count alike)

  if (warp == EM_GU_WARPS) {
    bool ok = true;
    // the next job at or after j that has rows in its tile
    const int both = p.sh_ff ? min(p.nff, p.sh_ff) : p.nff;  // rows that every segment has
    int e_n = 0, cnt_n = 0, off_n = 0;
    auto seek = [&](int j) {
      for (; j < n_jobs; j += gridDim.x) {
        const int seg = j / tiles_max, tile = j - seg * tiles_max;
        e_n = __ldcg(p.seg_expert + seg);
        cnt_n = __ldcg(p.seg_cnt + seg);
        off_n = __ldcg(p.seg_off + seg);
        if (tile * EM_FEAT < both || tile * EM_FEAT < (e_n >= p.n_expert ? p.sh_ff : p.nff)) break;
      }
      return j;
    };
    int pr_n = 0, row_n = 0;
    float xs_n = 0.f, wp_n = 1.f;
    auto pair_of = [&] { pr_n = (lane & 7) < cnt_n ? __ldcg(p.seg_pairs + off_n + (lane & 7)) : 0; };
    auto token_of = [&] {
      row_n = pr_n >= P ? pr_n - P : pr_n / p.n_used;
      xs_n = __ldcg(p.xscale + row_n);
      wp_n = (p.weight_before && e_n < p.n_expert) ? __ldcg(p.wts + pr_n) : 1.0f;
    };
    int job_n = seek(blockIdx.x);
    if (job_n < n_jobs) {
      pair_of();
      token_of();
    }
    for (int k = 0; ok; ++k) {
      const int job = job_n, e = e_n, cnt = cnt_n, pr = pr_n, row = row_n;
      const float xs = xs_n, wp = wp_n;
      const bool last = job >= n_jobs;
      const int seg = job / tiles_max, tile = job - seg * tiles_max;
      const bool shared_seg = e >= p.n_expert;
      const CUtensorMap* tmg = shared_seg ? &tm_sh_gate : &tm_gate;
      const CUtensorMap* tmu = shared_seg ? &tm_sh_up : &tm_up;
      const int bank_row0 = (shared_seg ? 0 : e * gu_rows) + tile * EM_FEAT;  // with gate and up in one bank the up map starts n_ff_exp rows in
      // lanes 8-23: a limb row of token (lane & 7); lanes 24-31: its sums.  A padding slot keeps what it held; its results are dropped.
      // In a narrow segment (see gateup_block) the high limbs follow the low ones four rows on.
      const bool mine = (lane & 7) < cnt;
      const uint32_t x_slot = lane < 16 ? lane - 8 : (cnt <= EM_NARROW ? EM_NARROW : 8) + (lane & 7);
      if (!last) job_n = seek(job + gridDim.x);
      for (int kc = 0; kc < n_kc; ++kc, ++it) {
        const int s = it % S;
        if (it >= (uint32_t)S && !mbar_wait_bounded(&s_empty[s], ((it / S) - 1) & 1)) { ok = false; break; }
        unsigned char* st = smem + (size_t)s * stage_bytes;
        if (kc == 0) {
          // free: with a stage of this job the consumers have left the job before last
          EmJob& d = s_job[k & 1];
          if (lane == 0) {
            d.job = last ? -1 : job;
            d.e = e;
            d.cnt = cnt;
          }
          if (lane < 8) {
            d.pair[lane] = pr;
            d.xs[lane] = xs;
            d.wp[lane] = wp;
          }
          __syncwarp();
          if (last) {
            if (lane == 0) mbar_arrive(&s_full[s]);
            break;
          }
        }
        if (lane == 0)
          mbar_arrive_expect_tx(&s_full[s], (uint32_t)(2 * EM_FEAT) * KB * Q4K_BLOCK_BYTES + (uint32_t)cnt * KB * (2 * 256 + 32));
        __syncwarp();
        if (lane < 2 * KB) {
          const int b = lane >> 1, role = lane & 1;
          tma_load_2d(st + (size_t)lane * BOX, role ? tmu : tmg, (kc * KB + b) * (int)Q4K_BLOCK_BYTES, bank_row0, &s_full[s]);
        } else if (lane >= 8 && lane < 24 && mine) {
          const int8_t* src = ((lane >= 16) ? p.xq_hi : p.xq_lo) + (size_t)row * p.ne + (size_t)kc * KB * 256;
          bulk_g2s(st + w_bytes + (size_t)x_slot * xpitch, src, (uint32_t)KB * 256, &s_full[s]);
        } else if (lane >= 24 && mine) {
          bulk_g2s(st + w_bytes + x_bytes + (size_t)(lane - 24) * spitch * 4, p.xsum + (size_t)row * nsb + (size_t)kc * KB * 8, (uint32_t)KB * 32, &s_full[s]);
        }
        if (kc == 0 && job_n < n_jobs) pair_of();
      }
      if (last) break;
      if (job_n < n_jobs) token_of();
    }
    if (!ok && lane == 0) atomicExch(&p.status->timeout, 7);
    return;
  }

  // consumers
  const int fw = warp & 1, ks = warp >> 1;
  int jpar = 0;
  bool ok = true;
  for (int k = 0; ok; ++k) {
    const EmJob& d = s_job[k & 1];
    bool narrow = false;
    float fg[4] = {0.f, 0.f, 0.f, 0.f}, fu[4] = {0.f, 0.f, 0.f, 0.f};
    for (int kc = 0; kc < n_kc; ++kc, ++it) {
      const int s = it % S;
      if (!mbar_wait_bounded(&s_full[s], (it / S) & 1)) { ok = false; break; }
      if (kc == 0) {
        if (d.job < 0) return;
        narrow = d.cnt <= EM_NARROW;
      }
      const unsigned char* st = smem + (size_t)s * stage_bytes;
      const unsigned char* wst = st + (size_t)(fw * 16 + g) * Q4K_BLOCK_BYTES;
      const unsigned char* x0 = st + w_bytes;
      const int* sums = reinterpret_cast<const int*>(st + w_bytes + x_bytes);
      for (int b = ks; b < KB; b += KS) {
        if (narrow)
          gateup_block<true>(wst + (size_t)b * 2 * BOX, BOX, x0 + (size_t)((g & 1) * EM_NARROW + (g >> 1)) * xpitch + 4 * t, 0, sums + (g >> 1) * spitch, b, fg, fu);
        else
          gateup_block<false>(wst + (size_t)b * 2 * BOX, BOX, x0 + (size_t)g * xpitch + 4 * t, (uint32_t)8 * xpitch, sums + g * spitch, b, fg, fu);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_empty[s]);  // (arrivals after the producer's last wait complete phases nobody waits for)
    }
    // the warps of a feature group add their sums up through two slots of shared memory (consumer warps only: named barrier 1).
    // Four: 2 and 3 onto 0 and 1, then 1 onto 0.  Two: the jobs take the slots in turn.
    if (!ok) s_abort = 1;
    auto put = [&](int slot) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        s_red[slot][fw][lane][i] = fg[i];
        s_red[slot][fw][lane][4 + i] = fu[i];
      }
    };
    auto add = [&](int slot) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        fg[i] += s_red[slot][fw][lane][i];
        fu[i] += s_red[slot][fw][lane][4 + i];
      }
    };
    auto meet = [] { asm volatile("bar.sync 1, %0;" ::"n"(EM_GU_WARPS * 32) : "memory"); };
    if (KS == 4 ? ks >= 2 : ks == 1) put(KS == 4 ? ks - 2 : jpar);
    meet();
    if (*reinterpret_cast<volatile int*>(&s_abort)) {
      ok = false;
      break;
    }
    if (KS == 4) {
      if (ks < 2) add(ks);
      if (ks == 1) put(1);  // (slot 1 was this warp's own to read)
      meet();
      if (ks == 0) add(1);
      meet();  // the slots are free for the next job
    } else {
      if (ks == 0) add(jpar);
      jpar ^= 1;
    }
    if (ks == 0) {
      // epilogue: act[pair, feature] = act_fn(gate) * up, f32
      const float clamp = d.e >= p.n_expert ? 0.f : p.clamp;
      const int f0 = d.job % tiles_max * EM_FEAT + fw * 16, cnt = d.cnt;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        // wide: rows g (i < 2) and g + 8 of tokens 2 t, 2 t + 1; narrow: rows g (i = 0) and g + 8 (i = 2) of token t
        const int tk = narrow ? t : 2 * t + (i & 1);
        if (tk >= cnt || (narrow && (i & 1))) continue;
        const float xs = d.xs[tk], wp = d.wp[tk];
        p.act[(size_t)d.pair[tk] * nffmax + f0 + g + 8 * (i >> 1)] = gated_act(p.act_kind, clamp, wp * (fg[i] * xs), wp * (fu[i] * xs));
      }
    }
  }
  if (!ok && lane == 0) atomicExch(&p.status->timeout, 7);
}

// ---------------------------------------------------------------------------------------------
// down
// ---------------------------------------------------------------------------------------------
// Four bytes of the 16-element sums of block b, K positions 4 t .. 4 t + 3 (`sums` is at the thread's own row and word).
__device__ __forceinline__ uint32_t sum_bytes(const unsigned char* sums, int b) { return *reinterpret_cast<const uint32_t*>(sums + 16 * b); }

// One 256-weight block of a warp's 16 output rows (rows g and g + 8) against the segment's tokens, added to acc (rows
// g: 0, 1; g + 8: 2, 3; wide: tokens 2t, 2t + 1; narrow: token t in 0 and 2).
//
// Q4_K: header (d, dmin, 12 scale bytes), then per 64 weights 32 code bytes whose low nibbles are the first 32-element
// group and high nibbles the second.
template <bool NARROW>
__device__ __forceinline__ void down_block_q4(const unsigned char* blk0, const unsigned char* blk1, const unsigned char* alo, const unsigned char* ahi,
                                              const unsigned char* sums, uint32_t sum_step, int b, float (&acc)[4]) {
  constexpr int NT = NARROW ? 1 : 2;
  const int t = threadIdx.x & 3;
  const unsigned char* blk[2] = {blk0, blk1};
  const uint4 hdr[2] = {*reinterpret_cast<const uint4*>(blk[0]), *reinterpret_cast<const uint4*>(blk[1])};
  int svl[2][NT], svh[2][NT], mv[2][NT];
  uint32_t scales[2][2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    q4k_scales(hdr[r].y, hdr[r].w, scales[r]);
#pragma unroll
    for (int k = 0; k < NT; ++k) svl[r][k] = svh[r][k] = 0;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t w0[2], w1[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      w0[r] = *reinterpret_cast<const uint32_t*>(blk[r] + 16 + 32 * j + 4 * t);       // k = 4 t .. 4 t + 3 of a group
      w1[r] = *reinterpret_cast<const uint32_t*>(blk[r] + 32 + 32 * j + 4 * t);       // k = 16 + 4 t ..
    }
#pragma unroll
    for (int hn = 0; hn < 2; ++hn) {
      const int k0 = b * 256 + j * 64 + hn * 32;
      const uint32_t a00 = (w0[0] >> (4 * hn)) & 0x0F0F0F0Fu, a10 = (w0[1] >> (4 * hn)) & 0x0F0F0F0Fu,
                     a01 = (w1[0] >> (4 * hn)) & 0x0F0F0F0Fu, a11 = (w1[1] >> (4 * hn)) & 0x0F0F0F0Fu;
      int cl[4] = {0, 0, 0, 0}, ch[4] = {0, 0, 0, 0};
      mma_u8s8_k32(cl, a00, a10, a01, a11, *reinterpret_cast<const uint32_t*>(alo + k0), *reinterpret_cast<const uint32_t*>(alo + k0 + 16));
      if (!NARROW) mma_u8s8_k32(ch, a00, a10, a01, a11, *reinterpret_cast<const uint32_t*>(ahi + k0), *reinterpret_cast<const uint32_t*>(ahi + k0 + 16));
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int sc = byte_of(scales[r][j >> 1], 2 * (j & 1) + hn);
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          svl[r][k] += sc * cl[2 * r + k];
          svh[r][k] += sc * (NARROW ? cl[2 * r + 1] : ch[2 * r + k]);
        }
      }
    }
  }
  {
    // K positions 4 t .. 4 t + 3 are the sums of 16 elements: a group's min stands twice
    uint32_t mins[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) mins[r] = __byte_perm(q4k_mins(hdr[r].z, hdr[r].w, t >> 1), 0, (t & 1) ? 0x3322 : 0x1100);
    offset_sums<NARROW, false>(mins[0], mins[1], sum_bytes(sums, b), NARROW ? 0u : sum_bytes(sums + sum_step, b), sum_bytes(sums + 2 * sum_step, b), mv[0], mv[1]);
  }
  // sum over the block of d sc sum(q X) - dmin m sum(X), X = 256 hi + lo
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const float d = f16_bits_to_f32(hdr[r].x), dmin = f16_bits_to_f32(hdr[r].x >> 16);
#pragma unroll
    for (int k = 0; k < NT; ++k)
      acc[2 * r + k] = fmaf(d, fmaf(256.f, (float)svh[r][k], (float)svl[r][k]), fmaf(-dmin, (float)mv[r][k], acc[2 * r + k]));
  }
}

// Byte `i` of w as a signed integer, by one byte permute that replicates the sign.
__device__ __forceinline__ int sext_byte(uint32_t w, int i) {
  uint32_t r;
  asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(w), "r"((uint32_t)(i * 0x1111) | 0x8880u));
  return (int)r;
}

// Q6_K: the slab starts on a 16-byte boundary, the rows' blocks at byte offsets ro0, ro1 on 2-byte ones.
template <bool NARROW>
__device__ __forceinline__ void down_block_q6(const unsigned char* slab, uint32_t ro0, uint32_t ro1, const unsigned char* alo, const unsigned char* ahi,
                                              const unsigned char* sums, uint32_t sum_step, int b, float (&acc)[4]) {
  constexpr int NT = NARROW ? 1 : 2;
  const int t = threadIdx.x & 3;
  // per row: aligned view of the block, the shift that realigns it, d and the 16 scales
  const uint32_t* wq[2];
  uint32_t sh[2];
  float d[2];
  uint32_t sc[2][4];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const uint32_t ro = r ? ro1 : ro0;
    sh[r] = (ro & 3u) * 8;
    wq[r] = reinterpret_cast<const uint32_t*>(slab + (ro & ~3u));
    d[r] = f16_bits_to_f32(*reinterpret_cast<const unsigned short*>(slab + ro + 208));
#pragma unroll
    for (int i = 0; i < 4; ++i) sc[r][i] = __funnelshift_r(wq[r][48 + i], wq[r][49 + i], sh[r]);
  }
  int svl[2][NT], svh[2][NT], mv[2][NT];
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int k = 0; k < NT; ++k) svl[r][k] = svh[r][k] = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
#pragma unroll
    for (int lh = 0; lh < 2; ++lh) {
      // words of ql (two 32-byte runs) and qh that hold l = 16 lh + 4 t .. + 3 of this half
      uint32_t A[2], B[2], H[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int o = 16 * h + 4 * lh + t;
        A[r] = __funnelshift_r(wq[r][o], wq[r][o + 1], sh[r]);
        B[r] = __funnelshift_r(wq[r][o + 8], wq[r][o + 9], sh[r]);
        const int oh = 32 + 8 * h + 4 * lh + t;
        H[r] = __funnelshift_r(wq[r][oh], wq[r][oh + 1], sh[r]);
      }
#pragma unroll
      for (int qd = 0; qd < 4; ++qd) {
        uint32_t a[2];
        int scv[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const uint32_t nib = (qd & 1) ? B[r] : A[r];
          a[r] = (((qd & 2) ? (nib >> 4) : nib) & 0x0F0F0F0Fu) | ((qd < 2 ? H[r] << (4 - 2 * qd) : H[r] >> (2 * qd - 4)) & 0x30303030u);
          const int si = 8 * h + 2 * qd + lh;  // scale index inside the block
          scv[r] = sext_byte(sc[r][si >> 2], si & 3);
        }
        const int k0 = b * 256 + h * 128 + qd * 32 + lh * 16;
        int cl[4] = {0, 0, 0, 0}, ch[4] = {0, 0, 0, 0};
        mma_u8s8_k16(cl, a[0], a[1], *reinterpret_cast<const uint32_t*>(alo + k0));
        if (!NARROW) mma_u8s8_k16(ch, a[0], a[1], *reinterpret_cast<const uint32_t*>(ahi + k0));
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int k = 0; k < NT; ++k) {
            svl[r][k] += scv[r] * cl[2 * r + k];
            svh[r][k] += scv[r] * (NARROW ? cl[2 * r + 1] : ch[2 * r + k]);
          }
      }
    }
  }
  {
    uint32_t own[2];  // the scales of K positions 4 t .. 4 t + 3
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const uint32_t even = (t & 2) ? sc[r][2] : sc[r][0], odd = (t & 2) ? sc[r][3] : sc[r][1];
      own[r] = (t & 1) ? odd : even;
    }
    offset_sums<NARROW, true>(own[0], own[1], sum_bytes(sums, b), NARROW ? 0u : sum_bytes(sums + sum_step, b), sum_bytes(sums + 2 * sum_step, b), mv[0], mv[1]);
  }
  // sum over the block of sc * (sum(q X) - 32 sum(X)), X = 256 hi + lo
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int k = 0; k < NT; ++k)
      acc[2 * r + k] = fmaf(d[r], fmaf(256.f, (float)svh[r][k], (float)svl[r][k]) - 32.f * (float)mv[r][k], acc[2 * r + k]);
}

// Job = (segment of up to 8 token rows, tile of `rows_cta` output features).  CTAs are persistent and take a
// contiguous range of jobs, so consecutive jobs mostly share their segment.  A job's rows are one contiguous
// slab of the expert's down matrix and arrive by one bulk copy into one of two buffers; the next job's slab
// is requested before this job is computed (the first one before the wait for the gate/up kernel).  When the
// segment changes, its activation rows are brought to 16-bit fixed point in shared memory (one scale per
// row, integer sums per 16 elements).  Q6_K blocks are 210 bytes, so a row's words sit 0 or 2 bytes off a
// word boundary: fragment words are two aligned loads and a funnel shift.  A 16-element scale group is one
// m16n8k16 MMA per limb; scales are applied in integers and converted once per block (bounded: 16 groups x
// 128 x 16 x 63 x 128 < 2^31).
// Q4 = the down banks are Q4_K (the other half of the layers of a Q4_K_M file): 144-byte blocks on 16-byte
// boundaries, so fragment words are plain loads; a 32-element scale group is one m16n8k32 MMA per limb, its
// 6-bit scale and min applied in integers (8 groups x 32 x 15 x 63 x 128 and 8 x 63 x 32 x 32639, both < 2^31).
// WARPS: 16 output rows per warp, or fewer rows (or more warps) and a split of the blocks over the warps.
// NBUF slab buffers.  The short jobs of four warps have one and, in the memory that this frees, more CTAs per SM to fill each
// other's waits (24 rows, Q6_K, 512 wide: 113 -> 107 us a layer; a scheduler then has 4.4 warps and still nothing to issue in
// 41 % of its cycles at 32 rows).  Eight warps have two (768 wide, 16 rows: 103 us against 115 with one) unless two leave room for 16 rows only:
// one of 32 then halves the jobs and their barriers (2048 wide, 64 rows: 1372 -> 1312 us).
// CTAs per SM asked of the compiler, as many as shared memory holds: left alone it takes 80 registers for eight warps of Q6_K, told of
// two CTAs 124, with more loads ahead of their use (128 experts of 1024, 32 rows: the layer 154 -> 148 us; of 768 121 -> 117), and of
// four warps 80 or 72 with spills instead of 96 or 80 (512 wide, the layer at 32 / 64 rows 108.4 / 137.3 -> 106.9 / 135.2, Q4_K at 32
// 74.7 -> 73.8).  Not for eight warps of Q4_K, of which three fit at 78 registers.
template <bool Q4, int WARPS, int NBUF>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 4 ? (Q4 ? 6 : 5) : Q4 ? 0 : 2) k_em_down(EmParams p, int rows_cta, int apitch, uint32_t slab_pitch) {
  constexpr uint32_t DBB = Q4 ? Q4K_BLOCK_BYTES : Q6K_BLOCK_BYTES;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t s_bar[2];
  __shared__ int s_pair[8];
  __shared__ float s_unit[8];  // a token's fixed-point unit
  __shared__ float s_dred[(WARPS - 1) * 128];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int tiles = p.ne / rows_cta;
  if (tid == 0) {
    mbar_init(&s_bar[0], 1);
    mbar_init(&s_bar[1], 1);
    mbar_fence_init();
  }
  __syncthreads();
  pdl_trigger();
  // the segment table is final (the gate/up kernel, ahead in the stream, only started after it)
  const int n_jobs = __ldcg(p.n_seg) * tiles;
  const int job0 = (int)((long long)blockIdx.x * n_jobs / gridDim.x), job1 = (int)((long long)(blockIdx.x + 1) * n_jobs / gridDim.x);
  if (job0 >= job1) return;
  const int sum_pitch = 16 * ((p.nffmax >> 8) | 1);  // bytes of a row of one byte of the sums: 4 (mod 8) words
  // shared memory: activation limbs [2][8 tokens][apitch] | bytes of the 16-element sums [3][8 tokens][sum_pitch] | NBUF slab buffers
  unsigned char* s_act = smem;
  unsigned char* s_sum = smem + (size_t)16 * apitch;
  unsigned char* slab_area = s_sum + 24 * sum_pitch;
  slab_area += (128u - (smem_u32(slab_area) & 127u)) & 127u;

  auto width_of = [&](int e) { return e >= p.n_expert ? p.sh_ff : p.nff; };
  auto src_of = [&](int e, int tile) {
    return (e >= p.n_expert ? p.sh_down : p.down + (size_t)e * p.down_stride) + (size_t)tile * rows_cta * (width_of(e) / 256 * (int)DBB);
  };
  // a slab lands at its source's offset inside a 128-byte line
  auto request = [&](int e, int tile, int buf) {
    const uint8_t* src = src_of(e, tile);
    const uint32_t bytes = (uint32_t)rows_cta * (width_of(e) / 256 * DBB);
    mbar_arrive_expect_tx(&s_bar[buf], bytes);
    bulk_g2s(slab_area + (size_t)buf * slab_pitch + (uint32_t)(reinterpret_cast<uintptr_t>(src) & 127u), src, bytes, &s_bar[buf]);
  };
  // segment table entries of the current segment and of the one after it, read a segment ahead
  int seg = job0 / tiles, tile = job0 - seg * tiles;
  const int last_seg = (job1 - 1) / tiles;
  int e = 0, cnt = 0, off = 0;
  int e_n = __ldcg(p.seg_expert + seg), cnt_n = __ldcg(p.seg_cnt + seg), off_n = __ldcg(p.seg_off + seg);
  if (tid == 0) request(e_n, tile, 0);
  bool fresh = true;
  int my_pair = tid < 8 && tid < cnt_n ? __ldcg(p.seg_pairs + off_n + tid) : -1;
  pdl_wait();  // activations come from the gate/up kernel

  for (int job = job0; job < job1; ++job, fresh = ++tile == tiles, seg += fresh, tile = fresh ? 0 : tile) {
    const int buf = NBUF == 2 ? (job - job0) & 1 : 0;
    if (fresh) {
      e = e_n;
      cnt = cnt_n;
      off = off_n;
      if (seg < last_seg) {
        e_n = __ldcg(p.seg_expert + seg + 1);
        cnt_n = __ldcg(p.seg_cnt + seg + 1);
        off_n = __ldcg(p.seg_off + seg + 1);
      }
    }
    const int nff_e = width_of(e);
    const unsigned char* slab = slab_area + (size_t)buf * slab_pitch + (uint32_t)(reinterpret_cast<uintptr_t>(src_of(e, tile)) & 127u);
    const int drb = nff_e / 256 * (int)DBB;
    __syncthreads();  // every warp is done with the previous job: its slab buffer (the other one) and the limbs may be reused
    if (NBUF == 2) {
      if (tid == 0 && job + 1 < job1) request(tile + 1 == tiles ? e_n : e, tile + 1 == tiles ? 0 : tile + 1, buf ^ 1);
    } else if (tid == 0 && job != job0) {
      request(e, tile, 0);
    }
    if (fresh) {
      if (job != job0) my_pair = tid < cnt ? __ldcg(p.seg_pairs + off + tid) : -1;
      if (tid < 8) s_pair[tid] = my_pair;
      __syncthreads();
      // fixed point: X = round(a * 32639 / max|a|) per row, limbs X = 256 hi + lo, sums per 16 elements.  A warp takes whole rows: no
      // barrier between a row's maximum and its rounding.  One unit per 128 elements, as in the per-pair kernels, has a little less
      // error (Q6_K, 13 rows of 512: 7.1e-5 of the result against 8.1e-5; Q4_K level) but costs two multiplications and a conversion
      // more for each of its results (Q4_K, 427 rows of 2560 over 512-wide experts: the kernel 76 us, 71 with one per row).  Another
      // unit also moves a layer's result by 6e-5, after which rows of a chain of layers now and then take another expert.
      const int n4 = nff_e / 4;
      for (int tk = warp; tk < cnt; tk += WARPS) {
        const float4* arow = reinterpret_cast<const float4*>(p.act + (size_t)s_pair[tk] * p.nffmax);
        auto top = [](float4 v, float m) { return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(m, fmaxf(fabsf(v.z), fabsf(v.w)))); };
        float inv = 0.f;
        auto unit = [&](float m) {
          m = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(m)));
          inv = m > 0.f ? 32639.f / m : 0.f;
          if (lane == 0) s_unit[tk] = m / 32639.f;
        };
        auto limbs = [&](int i, float4 v) {  // (n4 is a multiple of 64: whole warps)
          const int X[4] = {__float2int_rn(v.x * inv), __float2int_rn(v.y * inv), __float2int_rn(v.z * inv), __float2int_rn(v.w * inv)};
          uint32_t lo, hi;
          pack_limbs4(X, lo, hi);
          *reinterpret_cast<uint32_t*>(s_act + (size_t)tk * apitch + 4 * i) = lo;
          *reinterpret_cast<uint32_t*>(s_act + (size_t)((cnt <= EM_NARROW ? EM_NARROW : 8) + tk) * apitch + 4 * i) = hi;
          int sx = (X[0] + X[1]) + (X[2] + X[3]);  // 16 elements = four neighbouring lanes
          sx += __shfl_xor_sync(0xFFFFFFFFu, sx, 1);
          sx += __shfl_xor_sync(0xFFFFFFFFu, sx, 2);
          if ((i & 3) < 3) s_sum[((i & 3) * (cnt <= EM_NARROW ? EM_NARROW : 8) + tk) * sum_pitch + (i >> 2)] = (unsigned char)(sx >> (8 * (i & 3)));
        };
        float m = 0.f;
        if (n4 <= 128) {  // up to 512 wide: the row stays in registers
          float4 v[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) v[u] = lane + 32 * u < n4 ? __ldcg(arow + lane + 32 * u) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int u = 0; u < 4; ++u) m = top(v[u], m);
          unit(m);
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (lane + 32 * u < n4) limbs(lane + 32 * u, v[u]);
        } else {
#pragma unroll 4
          for (int i = lane; i < n4; i += 32) m = top(__ldcg(arow + i), m);
          unit(m);
#pragma unroll 4
          for (int i = lane; i < n4; i += 32) limbs(i, __ldcg(arow + i));
        }
      }
      __syncthreads();
    }
    if (!mbar_wait_bounded(&s_bar[buf], (NBUF == 2 ? (job - job0) >> 1 : job - job0) & 1)) {
      if (lane == 0) atomicExch(&p.status->timeout, 8);
      return;
    }
    const int nb = nff_e / 256;
    // 16-row tiles of this job: one per warp, or (fewer rows per CTA) several warps per tile, each taking
    // every ksplit-th block, their partial sums added through shared memory
    const int n_rt = rows_cta / 16, ksplit = WARPS / n_rt;
    // B fragments: wide - token g, limbs eight rows apart; narrow (see gateup_block) - limb g & 1 of token g / 2
    const bool narrow = cnt <= EM_NARROW;
    const unsigned char* alo = s_act + (size_t)(narrow ? (g & 1) * EM_NARROW + (g >> 1) : g) * apitch + 4 * t;
    const unsigned char* ahi = alo + (size_t)8 * apitch;
    // bytes of the sums: wide - of token g, byte k 8 k rows on; narrow - byte g & 1 of token g / 2, byte 2 eight rows on from byte 0's
    const uint32_t sum_step = (narrow ? EM_NARROW : 8) * sum_pitch;
    const unsigned char* sums = s_sum + (narrow ? (g & 1) * EM_NARROW + (g >> 1) : g) * sum_pitch + 4 * t;
    const int rt = warp % n_rt, ks = warp / n_rt;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    const uint32_t rofs[2] = {(uint32_t)(rt * 16 + g) * drb, (uint32_t)(rt * 16 + g + 8) * drb};
    for (int b = ks; b < nb; b += ksplit) {
      if (Q4 && narrow) down_block_q4<true>(slab + rofs[0] + (uint32_t)b * DBB, slab + rofs[1] + (uint32_t)b * DBB, alo, ahi, sums, sum_step, b, acc);
      if (Q4 && !narrow) down_block_q4<false>(slab + rofs[0] + (uint32_t)b * DBB, slab + rofs[1] + (uint32_t)b * DBB, alo, ahi, sums, sum_step, b, acc);
      if (!Q4 && narrow) down_block_q6<true>(slab, rofs[0] + (uint32_t)b * DBB, rofs[1] + (uint32_t)b * DBB, alo, ahi, sums, sum_step, b, acc);
      if (!Q4 && !narrow) down_block_q6<false>(slab, rofs[0] + (uint32_t)b * DBB, rofs[1] + (uint32_t)b * DBB, alo, ahi, sums, sum_step, b, acc);
    }
    if (ksplit > 1) {
      if (ks > 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) s_dred[((ks - 1) * n_rt + rt) * 128 + lane * 4 + i] = acc[i];
      }
      __syncthreads();
      if (ks == 0)
        for (int k2 = 1; k2 < ksplit; ++k2)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[i] += s_dred[((k2 - 1) * n_rt + rt) * 128 + lane * 4 + i];
    }
    // y[pair, row]: raw expert outputs; weights, down_scale and the sum over ranks follow in k_em_combine
    if (ks == 0) {
      const int i0 = tile * rows_cta + rt * 16;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int tk = narrow ? t : 2 * t + (i & 1);
        if (tk < cnt && !(narrow && (i & 1))) p.y[(size_t)s_pair[tk] * p.ne + i0 + g + 8 * (i >> 1)] = acc[i] * s_unit[tk];
      }
    }
  }
}

// dst[r, :] = sum over ranks (rank order) of w * (y[pair] * down_scale[e]), then the shared expert's row
// (sigmoid-gated when its logit is given), then the residual - the order of the per-pair kernels.
// A chain of three L2 reads behind the down kernel (8 us of 32 rows): the routing was complete before the down kernel started,
// so ids, weights and the residual are read while it still runs, and CTAs of 128 threads spread the rows over the device.
constexpr int EM_COMBINE_T = 128;
__global__ void __launch_bounds__(EM_COMBINE_T) k_em_combine(EmParams p, const float* sh_logit, const float* residual, float* dst) {
  const int c = (blockIdx.x * EM_COMBINE_T + threadIdx.x) * 4;
  if (c >= p.ne) return;
  const int P = p.rows * p.n_used;
  bool waited = false;
  for (int r = blockIdx.y; r < p.rows; r += gridDim.y) {
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f), h = o;
    if (residual != nullptr) h = __ldcg(reinterpret_cast<const float4*>(residual + (size_t)r * p.ne + c));  // may alias dst: each element is read, then written, by this thread
    const float gsh = (p.sh_ff && sh_logit) ? 1.0f / (1.0f + __expf(-__ldcg(sh_logit + r))) : 1.0f;
    for (int s0 = 0; s0 < p.n_used; s0 += 8) {
      // eight ranks at a time: ids and weights, then rows are requested together, then added in rank order
      float w[8], ds[8];
      bool on[8];
      float4 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int pr = r * p.n_used + s0 + j;
        const bool in = s0 + j < p.n_used;
        int e = in ? __ldcg(p.ids + pr) : -1;
        on[j] = e >= 0;
        e = min(e, p.n_expert - 1);
        if (p.ep_n != 0 && ((uint32_t)e < p.ep_lo || (uint32_t)e >= p.ep_lo + p.ep_n)) on[j] = false;
        ds[j] = (on[j] && p.down_scale) ? __ldg(p.down_scale + e) : 1.0f;
        w[j] = on[j] ? (p.weight_before ? 1.0f : __ldcg(p.wts + pr)) : 0.f;
      }
      if (!waited) {
        pdl_wait();  // the rows come from the down kernel
        waited = true;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[j] = on[j] ? __ldcg(reinterpret_cast<const float4*>(p.y + (size_t)(r * p.n_used + s0 + j) * p.ne + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {  // a skipped rank adds 0 * 0: the sum is the one over the served ranks, in order
        v[j].x *= ds[j]; v[j].y *= ds[j]; v[j].z *= ds[j]; v[j].w *= ds[j];
        o.x += w[j] * v[j].x; o.y += w[j] * v[j].y; o.z += w[j] * v[j].z; o.w += w[j] * v[j].w;
      }
    }
    if (p.sh_ff) {
      const float4 v = __ldcg(reinterpret_cast<const float4*>(p.y + (size_t)(P + r) * p.ne + c));
      o.x += gsh * v.x; o.y += gsh * v.y; o.z += gsh * v.z; o.w += gsh * v.w;
    }
    if (residual != nullptr) {
      o.x += h.x; o.y += h.y; o.z += h.z; o.w += h.w;
    }
    *reinterpret_cast<float4*>(dst + (size_t)r * p.ne + c) = o;
  }
}

// Stage shape of the gate/up kernel: KB blocks of every row per stage (even where the row allows it: the
// two block-parity warps then share a stage evenly), S stages, two CTAs per SM.
void gateup_shape(int ne, int* KB, int* S, int* xpitch, size_t* stage_bytes) {
  const int nblk = ne / 256;
  const int kb = (nblk % 4 == 0) ? 4 : ((nblk % 2 == 0) ? 2 : 1);
  *xpitch = kb * 256 + 16;  // 4 (mod 32) words
  *stage_bytes = (size_t)kb * 2 * EM_FEAT * Q4K_BLOCK_BYTES + (size_t)16 * *xpitch + (size_t)8 * (kb * 8 + 4) * 4;
  int s = nblk / kb;
  while (s > 1 && (s > EM_MAX_STAGES || (size_t)s * *stage_bytes > 112 * 1024)) --s;
  *KB = kb;
  *S = s;
}

// Rows of the down matrix per job: 64 (one 16-row tile per warp) while the slab buffers and the activation
// limbs leave room for two CTAs per SM, else 32 or 16 with the blocks split over the warps.
// Eight warps where a row has at least three blocks to split (64 rows, 28 MB experts: the layer 1511 -> 1384 us), four for
// shorter rows, whose jobs the extra barrier costs more than it gives (32 rows, 512-wide experts: 153 -> 168 us).
int down_warps(int nffmax) { return nffmax >= 768 ? 8 : 4; }

using DownKernel = void (*)(EmParams, int, int, uint32_t);

struct DownShape {
  int rows, apitch, nbuf, warps;  // rows 0: no tile fits shared memory
  size_t slab_pitch, smem;
  DownKernel kernel;
};

DownShape down_shape(int ne, int nffmax, bool q4k) {
  DownShape d = {};
  d.apitch = nffmax + 16;  // 4 (mod 32) words
  const size_t dbb = q4k ? Q4K_BLOCK_BYTES : Q6K_BLOCK_BYTES;
  const size_t fixed = (size_t)16 * d.apitch + (size_t)8 * (nffmax / 16 + 4) * 4 + 256;  // limbs, sums (with room to spare)
  const size_t drb = (size_t)nffmax / 256 * dbb;
  const int nb = nffmax / 256;
  d.warps = down_warps(nffmax);
  const int most = d.warps == 8 ? 2 : 1;
  auto choose = [&]() {
    for (int rows : {64, 32, 16}) {
      if (ne % rows) continue;
      if (nb == 1 && rows < 64) continue;  // (fewer rows only spread the blocks over more warps)
      d.slab_pitch = align_up((size_t)rows * drb + 8, 128) + 128;
      for (d.nbuf = most; d.nbuf >= 1; --d.nbuf) {
        d.smem = fixed + d.nbuf * d.slab_pitch;
        if (rows == 16) return d.smem <= 200 * 1024 ? rows : 0;
        if (d.smem <= 110 * 1024) return rows;
        if (rows != 32) break;
      }
    }
    return 0;
  };
  d.rows = choose();
  if (d.warps == 4)
    d.kernel = q4k ? k_em_down<true, 4, 1> : k_em_down<false, 4, 1>;
  else if (d.nbuf == 2)
    d.kernel = q4k ? k_em_down<true, 8, 2> : k_em_down<false, 8, 2>;
  else
    d.kernel = q4k ? k_em_down<true, 8, 1> : k_em_down<false, 8, 1>;
  return d;
}

}  // namespace

size_t em_scratch_bytes(int rows, int n_used, int ne, int nff, int sh_ff) {
  const size_t PT = (size_t)rows * n_used + rows, nffmax = std::max(nff, sh_ff);
  const size_t max_seg = PT + 8;
  size_t b = 0;
  b += align_up((size_t)rows * (ne / 32) * 4, 256);     // xsum
  b += align_up(256, 256);                              // n_seg
  b += 3 * align_up(max_seg * 4, 256);                  // seg_expert, seg_off, seg_cnt
  b += align_up((PT + 8) * 4, 256);                     // seg_pairs
  b += align_up(PT * nffmax * 4, 256);                  // act
  b += align_up(PT * (size_t)ne * 4, 256);              // y
  return b;
}

bool em_supported(int ne, int nff, int sh_ff, int n_expert, BankTypes bt) {
  if (!bt.tuned() || ne % 256 || nff % 256 || sh_ff % 256 || n_expert > 1024) return false;
  return down_shape(ne, std::max(nff, sh_ff), bt.down_q4k()).rows != 0;
}

int em_down_ctas_per_sm(int ne, int nff, int sh_ff, bool q4k) {
  const DownShape d = down_shape(ne, std::max(nff, sh_ff), q4k);
  int n = 0;
  return d.rows != 0 && resident_ctas(reinterpret_cast<const void*>(d.kernel), d.warps * 32, d.smem, &n) == cudaSuccess ? n : 0;
}

int32_t launch_em_ffn(infr_cuda_ctx* ctx, const DecodeParams& dp, void* scratch, uint32_t stages) {
  EmParams p = {};
  const int rows = dp.rows, P = rows * dp.n_used, sh_ff = dp.sh_gate ? dp.sh_ff : 0;
  const size_t PT = (size_t)P + rows, nffmax = std::max(dp.nff, sh_ff), max_seg = PT + 8;
  char* base = static_cast<char*>(scratch);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* q = base + off;
    off += align_up(bytes, 256);
    return q;
  };
  p.xsum = reinterpret_cast<int*>(take((size_t)rows * (dp.ne / 32) * 4));
  p.n_seg = reinterpret_cast<int*>(take(256));
  p.seg_expert = reinterpret_cast<int*>(take(max_seg * 4));
  p.seg_off = reinterpret_cast<int*>(take(max_seg * 4));
  p.seg_cnt = reinterpret_cast<int*>(take(max_seg * 4));
  p.seg_pairs = reinterpret_cast<int*>(take((PT + 8) * 4));
  p.act = reinterpret_cast<float*>(take(PT * nffmax * 4));
  p.y = reinterpret_cast<float*>(take(PT * (size_t)dp.ne * 4));
  p.xsum_ready = dp.xsum_ready;
  p.xq_lo = dp.xq_lo;
  p.xq_hi = dp.xq_hi;
  p.xscale = dp.xscale;
  p.ids = dp.ids;
  p.wts = dp.wts;
  p.gate = dp.gate; p.up = dp.up; p.down = dp.down;
  p.sh_gate = dp.sh_gate; p.sh_up = dp.sh_up; p.sh_down = dp.sh_down;
  p.gate_stride = dp.gate_stride; p.up_stride = dp.up_stride; p.down_stride = dp.down_stride;
  p.down_scale = dp.down_scale;
  p.status = dp.status;
  p.rows = rows; p.ne = dp.ne; p.n_used = dp.n_used; p.nff = dp.nff; p.sh_ff = sh_ff; p.n_expert = dp.n_expert;
  p.nffmax = (int)nffmax;
  p.ep_lo = dp.ep_lo; p.ep_n = dp.ep_n;
  p.act_kind = dp.act_kind; p.weight_before = dp.weight_before; p.clamp = dp.clamp;

  // segments: one per expert with pairs, plus one per further EM_SEG pairs of an expert, plus the shared expert's
  const int max_routed_seg = std::min(P, dp.n_expert) + P / EM_SEG;
  const int n_seg_bound = max_routed_seg + (sh_ff ? (rows + EM_SEG - 1) / EM_SEG : 0);
  cudaError_t e = cudaSuccess;
  if (stages & 2u) {
    e = launch_ex(k_em_bucket, dim3(1), dim3(1024), 0, ctx->stream, true, p, EM_SEG);
    ctx->launches += 1;
    if (e != cudaSuccess) return check_cuda(ctx, e, "k_em_bucket launch");
    int KB, S, xpitch;
    size_t stage_bytes;
    gateup_shape(dp.ne, &KB, &S, &xpitch, &stage_bytes);
    const size_t smem = (size_t)S * stage_bytes;
    // the banks' rows as 2-D tensors for the tiled copies; with gate and up in one bank an expert has
    // 2 n_ff_exp rows and the up map starts n_ff_exp rows in (and ends with the bank)
    const size_t rb = (size_t)dp.ne / 256 * Q4K_BLOCK_BYTES;
    const size_t rows_per_expert = dp.gate_stride / rb, bank_rows = (size_t)dp.n_expert * rows_per_expert;
    CUtensorMap tm_gate, tm_up, tm_sh_gate, tm_sh_up;
    bool ok = q4k_rows_map(&tm_gate, dp.gate, bank_rows, rb, EM_FEAT) &&
              q4k_rows_map(&tm_up, dp.up, bank_rows - (rows_per_expert - (size_t)dp.nff), rb, EM_FEAT);
    tm_sh_gate = tm_gate;
    tm_sh_up = tm_up;
    if (ok && sh_ff) ok = q4k_rows_map(&tm_sh_gate, dp.sh_gate, (size_t)sh_ff, rb, EM_FEAT) && q4k_rows_map(&tm_sh_up, dp.sh_up, (size_t)sh_ff, rb, EM_FEAT);
    if (!ok) return fail(ctx, INFR_CUDA_ERR_CUDA, "expert-major gate/up kernel: the driver refused a tensor map for the expert banks");
    // persistent CTAs: two per SM (the shared-memory request allows no more), never more than there are jobs
    const unsigned jobs_bound = (unsigned)n_seg_bound * (unsigned)(nffmax / EM_FEAT);
    auto run_gu = [&](auto kern, unsigned threads) {
      cudaError_t ee = ensure_smem(reinterpret_cast<const void*>(kern), smem);
      if (ee == cudaSuccess)
        ee = launch_ex(kern, dim3(std::min(jobs_bound, 2u * (unsigned)ctx->sm_count)), dim3(threads), smem, ctx->stream, true, p, KB, S, xpitch,
                       (int)rows_per_expert, tm_gate, tm_up, tm_sh_gate, tm_sh_up);
      return ee;
    };
    // A long row keeps four warps per feature group busy and hides the tree of sums at its end (7168 wide, 64 rows: 1511 us a
    // layer with two, 1384 with four); rows of 8 blocks are done too soon for it (2048 wide, 32 rows: 152 against 153 us).
    e = dp.ne >= 4096 ? run_gu(k_em_gateup<4>, 9 * 32) : run_gu(k_em_gateup<2>, 5 * 32);
    ctx->launches += 1;
    if (e != cudaSuccess) return check_cuda(ctx, e, "k_em_gateup launch");
  }
  if (!(stages & 4u)) return INFR_CUDA_OK;
  {
    const DownShape d = down_shape(dp.ne, (int)nffmax, dp.down_q4k != 0);
    if (!d.rows) return fail(ctx, INFR_CUDA_ERR_UNSUPPORTED, "expert-major down kernel: tile does not fit shared memory");
    const unsigned jobs_bound = (unsigned)n_seg_bound * (unsigned)(dp.ne / d.rows);
    // as many CTAs as an SM holds of them: with fewer, SMs are half used, or idle where two of a grid's CTAs land on one; with more,
    // the last ones, whose share of the jobs is as large as the others', run behind them.  Asked of the driver: by 215 KB over the
    // request + 3 KB it was two of three (Q4_K, 128 experts of 1280, 32 rows: the layer 179 -> 157 us; of 768 116 -> 105), one of two
    // (Q6_K, 1536: 274 -> 203) and six of five (Q6_K, 256: 65.4 -> 61.5)
    int per_sm = 0;
    e = resident_ctas(reinterpret_cast<const void*>(d.kernel), d.warps * 32, d.smem, &per_sm);
    if (e == cudaSuccess)
      e = launch_ex(d.kernel, dim3(std::min(jobs_bound, (unsigned)(per_sm * ctx->sm_count))), dim3(d.warps * 32), d.smem, ctx->stream, true, p,
                    d.rows, d.apitch, (uint32_t)d.slab_pitch);
    ctx->launches += 1;
    if (e != cudaSuccess) return check_cuda(ctx, e, "k_em_down launch");
  }
  e = launch_ex(k_em_combine, dim3((dp.ne / 4 + EM_COMBINE_T - 1) / EM_COMBINE_T, std::min(rows, 65535)), dim3(EM_COMBINE_T), 0, ctx->stream, true, p, dp.sh_logit,
                dp.residual, dp.dst);
  ctx->launches += 1;
  return check_cuda(ctx, e, "k_em_combine launch");
}

}  // namespace infr

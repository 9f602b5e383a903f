// Shapes of the per-pair kernels' launches (decode_ffn.cu): plain host arithmetic.
#pragma once
#include <algorithm>
#include <cstddef>

namespace infr {

constexpr int GU_WARPS = 16;  // rows per chunk and role: one per warp
constexpr int GU_MAX_CHUNKS = 4;
constexpr int GU_XQPITCH = 144;  // bytes per 64-element group of fixed-point x: 64 low limbs, 64 high limbs, pad

inline size_t gateup_smem(int ne, int n_chunks, size_t gbb, int gw = GU_WARPS) {
  return (size_t)n_chunks * 2 * gw * (ne / 256 * gbb) + (size_t)(ne / 64) * GU_XQPITCH;
}

// Chunks per CTA for gate/up banks of gbb bytes per block, 0 where none fit.
inline int pick_chunks(int ne, int nff, int sh_ff, size_t gbb) {
  for (int c = 2; c >= 1; c >>= 1) {
    const int TR = GU_WARPS * c;
    if (nff % TR) continue;
    if (sh_ff && sh_ff % TR) continue;
    if (gateup_smem(ne, c, gbb) <= 200 * 1024) return c;
  }
  return 0;
}

struct GateUpShape {
  int warps, chunks, ctas;
};

// The shape a launch takes; ew, ec: infr_cuda_config::gu_warps and gu_chunks.
//
// One wave (a CTA to an SM): 16 warps x 2 chunks, x 1 while even half as many would do with Q4_K (1024 wide, 32 experts of 256, one
// row: 12.4 -> 11.2 us the layer).
// More: smaller CTAs put more independent chains of (ids -> copies -> unpack) on an SM.  Up to two waves 8 x 2, then 4 x 2 where
// four warps stage a row's limbs (2048 wide), else 8 x 2; past four waves the config's (4 x 4: 69 us against 78 for 32 tokens), these where
// the config's does not fit the dims, and the one-wave shape where the config says so.  us the layer, 16 x 2 / 8 x 2 / 4 x 2:
// 2048 wide, 256 of 512, Q4_K: two rows 22.5 / 22.6 / 23.2, four 37.7 / 37.2 / 36.9; Q5_K: two 26.3 / 25.3 / 24.9, four 45.4 / 41.4 / 40.7;
// 4096 wide, 1024: one row 28.0 / 25.3, four 73.3 / 70.1; 3072 wide, 512: two rows 26.7 / 23.0, eight 73.8 / 64.8.
inline GateUpShape gateup_shape(int ne, int nff, int sh_ff, int rows, int n_used, size_t gbb, bool q5k, int sms, int ew,
                                int ec) {
  GateUpShape s = {GU_WARPS, std::max(pick_chunks(ne, nff, sh_ff, gbb), 1), 0};
  auto ctas = [&](int tr) { return rows * n_used * (nff / tr) + rows * (sh_ff / tr); };
  auto take = [&](int w, int c) {  // w warps, c chunks: enough threads for the limbs of a row, whole tiles
    if (ne / 16 > w * 32 || nff % (w * c) || sh_ff % (w * c) || gateup_smem(ne, c, gbb, w) > 200 * 1024) return false;
    s = {w, c, ctas(w * c)};
    return true;
  };
  const int full = s.ctas = ctas(s.warps * s.chunks);
  if (full <= sms) {
    if (!q5k && s.chunks == 2 && 2 * full <= sms) take(GU_WARPS, 1);
    return s;
  }
  if (full > 4 * sms) {
    if (ew == 0 || ec == 0) return s;
    if (take(ew, ec)) return s;
  }
  if (!(full > 2 * sms && take(4, 2))) take(8, 2);
  return s;
}

constexpr int DN_MAX_WARPS = 24;

// Warps of a down CTA.  Its time is a chain of latencies (activations read and rounded by all warps, a task of up to eight rows of a
// slot per warp), so a CTA takes the warps that its SM's registers leave it: an SM holds 36 warps of these registers.
// fit: CTAs that an SM's shared memory holds, as the driver has it (two of 114 KB: 2560 wide, six 1024-wide slots and a shared one, Q6_K, one /
// three rows 24.8 / 47.5 us the layer, 29.0 / 56.1 where a bound with room to spare said one).
//   grid of one wave: 20, which fit beside a gate/up CTA of 16 (128 experts of 768, one row: 16 warps 20.0 us the layer, 20 18.6);
//   shared memory holds one CTA only: all 24 (7168 wide, 2048, one row: 9 warps 158 us, 24 132);
//   past four waves: a divisor of the tasks under the cap (infr_cuda_config::dn_warps; 32 rows: 83 us with three CTAs of 12 to an SM,
//   98 with two of 16), or the cap itself where that leaves fewer than nine and tasks are heavy or two CTAs fit (16 tasks of Q6_K, six rows:
//   8 warps 65.2 us, 12 63.5; 14 tasks, two fit, eight rows 124 / 120, Q4_K 120 / 115; but of Q4_K with more to an SM 7 warps 52.3, 12 56.3);
//   else as many CTAs share an SM as the grid has for it and shared memory and a task per warp allow, fewer where that takes no
//   wave more and a round of tasks less (16 tasks of Q4_K, 512 CTAs: three of 8 warps 48.7, two of 16 46.9).  Q4_K, whose tasks are lighter:
//   whole rounds of tasks where there are several waves.  256 experts of 512: three rows 18 warps 32.2 us, 12 30.0; Q4_K down, three rows
//   30.8 / 28.1, four rows 18 warps 35.2, 12 35.5, 9 32.3; two 768-wide slots and a shared one, two rows 6 warps 19.9, 18 16.6.
// Over 280 launches (18 layers, one to twelve rows, both formats) this is 1.4 % over the best count of warps for each, and 9 % at most.
inline int down_warps(int ctas, int n_tasks, int fit, bool q4k, int sms, int cap) {
  if (ctas <= sms) return 20;
  if (fit <= 1) return DN_MAX_WARPS;
  if (ctas > 4 * sms && cap > 0) {
    int c = std::min(cap, n_tasks);
    while (n_tasks % c) --c;
    return c < 9 && n_tasks > cap && (!q4k || fit == 2) ? cap : c;
  }
  int k = std::min(std::min((ctas + sms - 1) / sms, fit), 36 / std::min(std::max(n_tasks, 6), 9));
  auto waves = [&](int n) { return (ctas + n * sms - 1) / (n * sms); };
  auto rounds = [&](int n) { return (n_tasks + 36 / n - 1) / (36 / n); };
  while (k > 2 && waves(k - 1) == waves(k) && rounds(k - 1) < rounds(k)) --k;
  if (q4k && k > 2 && waves(k) > 1) return (n_tasks + rounds(k) - 1) / rounds(k);
  const int nw = 36 / k;
  if (k >= 4) return std::min(nw, std::max(n_tasks, 6));
  return k == 2 && n_tasks >= 14 ? std::min(nw, n_tasks) : nw;
}

}  // namespace infr

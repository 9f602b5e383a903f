// CTAs of the per-pair gate/up kernel (decode_ffn.cu): plain host arithmetic.
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

}  // namespace infr

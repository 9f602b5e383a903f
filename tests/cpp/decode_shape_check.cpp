// Prints the shape (warps, row chunks, CTAs) of a per-pair gate/up launch: ne nff sh_ff rows n_used block_bytes q5k sms gu_warps gu_chunks
// or the warps of a down launch's CTA: ctas tasks fit q4k sms dn_warps
#include <cstdio>
#include <cstdlib>

#include "decode_shape.h"

int main(int argc, char** argv) {
  int v[10];
  for (int i = 0; i < argc - 1 && i < 10; ++i) v[i] = std::atoi(argv[i + 1]);
  if (argc == 7) {
    std::printf("%d\n", infr::down_warps(v[0], v[1], v[2], v[3] != 0, v[4], v[5]));
    return 0;
  }
  if (argc != 11) return 2;
  const infr::GateUpShape s = infr::gateup_shape(v[0], v[1], v[2], v[3], v[4], v[5], v[6] != 0, v[7], v[8], v[9]);
  std::printf("%d %d %d\n", s.warps, s.chunks, s.ctas);
  return 0;
}

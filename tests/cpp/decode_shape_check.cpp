// Prints the shape (warps, row chunks, CTAs) of a per-pair gate/up launch: ne nff sh_ff rows n_used block_bytes q5k sms gu_warps gu_chunks
#include <cstdio>
#include <cstdlib>

#include "decode_shape.h"

int main(int argc, char** argv) {
  if (argc != 11) return 2;
  int v[10];
  for (int i = 0; i < 10; ++i) v[i] = std::atoi(argv[i + 1]);
  const infr::GateUpShape s = infr::gateup_shape(v[0], v[1], v[2], v[3], v[4], v[5], v[6] != 0, v[7], v[8], v[9]);
  std::printf("%d %d %d\n", s.warps, s.chunks, s.ctas);
  return 0;
}

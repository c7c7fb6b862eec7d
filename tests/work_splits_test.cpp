// Host cases of csrc/splits.h: how the kernels deal their work.
#include <cstdio>

#include "splits.h"

static int fail(const char* what, int a, int b) { std::printf("%s: %d %d\n", what, a, b); return 1; }

// The cluster's selection: shares cover the row in order, differ by one element at most, and hold at least 512 elements of any row whose
// elements do not all fit the candidate list (4,096): 16 warps of 32, whose four best make the 64 that a CTA has to offer.
static int topk_shares() {
  for (int nb = 513; nb <= 262144; ++nb) {
    if (cr::topk_share(nb, 0) != 0 || cr::topk_share(nb, 8) != nb) return fail("topk_share ends", nb, cr::topk_share(nb, 8));
    for (int k = 0; k < 8; ++k) {
      const int n = cr::topk_share(nb, k + 1) - cr::topk_share(nb, k);
      if (n < nb / 8 || n > (nb + 7) / 8) return fail("topk_share uneven", nb, n);
      if (nb > 4096 && n < 512) return fail("topk_share short", nb, n);
      if (n > (nb <= 65536 ? 8 : 32) * 1024) return fail("topk_share above the registers", nb, n);
    }
  }
  return 0;
}

// The tiles of a launch of span scores: no CTA is left for a second wave, and no warp walks more tiles than that takes.
static int score_tiles() {
  for (int sms = 132; sms <= 160; sms += 16)
    for (int n = 1; n <= 32; ++n)
      for (int tiles = 16; tiles <= 8192; ++tiles) {
        const int per = cr::score_tiles_per_warp(tiles, n, sms);
        auto ctas = [&](int p) { return n * ((tiles + 4 * p - 1) / (4 * p)); };
        if (per < 1 || ctas(per) > 3 * sms) return fail("score_tiles_per_warp: a second wave", tiles, n);
        if (per > 1 && ctas(per - 1) <= 3 * sms) return fail("score_tiles_per_warp: more than needed", tiles, n);
      }
  return 0;
}

int main() {
  if (topk_shares() || score_tiles()) return 1;
  std::puts("work_splits_test: ok");
  return 0;
}

// How work is dealt to CTAs, in plain C++: the launchers and kernels share it with the host tests.
#pragma once
#if defined(__CUDACC__)
#define CR_SPLIT __host__ __device__ constexpr
#else
#define CR_SPLIT constexpr
#endif

namespace cr {

// First element of CTA `rank` of the eight that select from a row of `count` blocks together (its share ends where the next begins).
CR_SPLIT int topk_share(int count, int rank) { return (int)((long long)count * rank / 8); }

// Pool tiles that a warp walks, so that the CTAs of four warps of all `n` spans (as many for each as the longest needs, which has
// `tiles`) run at once, three to an SM.
CR_SPLIT int score_tiles_per_warp(int tiles, int n, int sms) {
  const int ctas = 3 * sms / n > 0 ? 3 * sms / n : 1;                  // of a span
  return (tiles + 4 * ctas - 1) / (4 * ctas);
}

}  // namespace cr

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

}  // namespace cr

// Indexer scores of short spans (3..16 rows: verify passes, short decode batches) as an HBM stream through
// mma.sync: the job of QsaScoreRowsKernel (engine/layers/qsa_long.h:44-108) for spans too long for the one-row stream
// (qsa_score4_kernel) and too short to fill the 128-row tiles of the tcgen05 kernel (qsa_score_tc.cu).
//
// The pool tile [128 dims][32 blocks] fp32 is, as it lies in HBM, the "column" operand of m16n8k16: a thread's B
// fragments are pool[d][b] for four dims and, as columns of four products, four blocks, so every load instruction of a warp is
// four full lines and nothing is transposed or staged.  Rows of the product are (row, indexer head) pairs, m = 4 r + h, so the
// four heads of a row sit in four neighbouring lanes and relu + sum is two exchanges.  Queries and pool values are split
// into fp16 head + remainder (hi hi + lo hi + hi lo, fp32 accumulation): scores agree with fp32 dot products to 1e-5.
// One warp owns whole tiles and walks them in steps of 16 dims; the loads of three steps are in flight ahead of the one
// that multiplies, the first ones while the queries are staged.
//
// Bound: latency with ten to twelve warps on an SM (tensor pipe 49 %, shared memory and L1 56 % busy).  With half a tile a step in
// 4-byte loads (128 of four lines and 96 ldmatrix a tile) and four tiles to a warp whatever their number, 8 sessions x 9 rows
// at 131,072 took 52 us and one session x 4 rows at 32,003 (16 CTAs) 14.4; 37 and 5.5 us now.
#include <type_traits>
#include "qsa.cuh"
#include "splits.h"

namespace cr {

constexpr int kSmLd = 136;                   // halves per query row in shared memory (272 bytes: conflict-free ldmatrix)

__device__ __forceinline__ void sm_ldsm_x4(unsigned (&r)[4], const void* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void sm_mma(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// (x, y) as fp16 pair and the fp16 pair of what the rounding lost
__device__ __forceinline__ void split_pair(float x, float y, unsigned& hi, unsigned& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 b = __half22float2(h);
  const __half2 r = __floats2half2_rn(x - b.x, y - b.y);
  hi = *reinterpret_cast<const unsigned*>(&h);
  lo = *reinterpret_cast<const unsigned*>(&r);
}

// Four blocks' values of a dim.  Pools off the 16-byte boundary (!WIDE, some pool of the launch) are read a float at a time.
template <bool WIDE>
__device__ __forceinline__ float4 sm_load4(const float* p) {
  if constexpr (WIDE) return __ldcg(reinterpret_cast<const float4*>(p));
  else return make_float4(p[0], p[1], p[2], p[3]);
}

// grid (tile groups, 1, spans), 128 threads; MT = ceil(rows / 4) m-tiles of 16 (row, head) pairs; a warp walks `per_warp` tiles.
template <int MT, bool WIDE>
__global__ void __launch_bounds__(128, 3) qsa_score_mma_kernel(const __grid_constant__ QsaParams P, int per_warp) {
  const cr_qsa_args& a = P.span[blockIdx.z];
  pdl_release();
  const int nb_all = (a.pos0 + a.R) / 4;              // blocks complete for the last row
  __shared__ __align__(16) __half qh[16 * MT][kSmLd], ql[16 * MT][kSmLd];
  const int t = threadIdx.x, w = t >> 5, l = t & 31, g = l >> 2, tq = l & 3;
  const int tiles = (nb_all + 31) / 32;
  const int first = (blockIdx.x * 4 + w) * per_warp, last = min(first + per_warp, tiles);
  const bool scored = nb_all > CR_SEL_BLOCKS && a.R <= 4 * MT;
  touch_params(a);
  pdl_wait();
  if (!scored) return;
  // A step is 16 dims of a whole tile: this thread's four 16-byte loads are the dims 16 ks + 2 tq + {0, 1, 8, 9} of the blocks
  // 4 g .. 4 g + 3, and block 4 g + nt is column g of product nt.  Three steps are in flight ahead of the one in use.
  const int total = (last - first) * 8;
  const float* pt = a.c.ik_pool + (size_t)first * 4096 + 2 * tq * 32 + 4 * g;
  auto fetch = [&](float4 (&v)[4], int step) {
    const float* p = pt + (size_t)step * 512;          // tiles lie back to back
    v[0] = sm_load4<WIDE>(p); v[1] = sm_load4<WIDE>(p + 32); v[2] = sm_load4<WIDE>(p + 256); v[3] = sm_load4<WIDE>(p + 288);
  };
  float4 ring[4][4];
  if (first < last) { fetch(ring[0], 0); fetch(ring[1], 1); fetch(ring[2], 2); }   // in flight while the queries are staged; total >= 8
  for (int i = t; i < 16 * MT * 64; i += 128) {        // pairs of dims: row m = 4 r + h of the span's normalised indexer queries
    const int m = i >> 6, d = (i & 63) * 2, r = m >> 2, h = m & 3;
    float2 v = make_float2(0.f, 0.f);
    if (r < a.R) v = *reinterpret_cast<const float2*>(a.idx + (size_t)r * 640 + h * 128 + d);
    unsigned hi, lo;
    split_pair(v.x, v.y, hi, lo);
    *reinterpret_cast<unsigned*>(&qh[m][d]) = hi;
    *reinterpret_cast<unsigned*>(&ql[m][d]) = lo;
  }
  __syncthreads();
  if (first >= last) return;
  for (int s0 = 0; s0 < total; s0 += 8) {
    float acc[MT][4][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) acc[m][nt][0] = acc[m][nt][1] = acc[m][nt][2] = acc[m][nt][3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      if (s0 + ks + 3 < total) fetch(ring[(ks + 3) & 3], s0 + ks + 3);
      const float4 (&v)[4] = ring[ks & 3];
      unsigned bh[4][2], bl[4][2];
      split_pair(v[0].x, v[1].x, bh[0][0], bl[0][0]); split_pair(v[2].x, v[3].x, bh[0][1], bl[0][1]);
      split_pair(v[0].y, v[1].y, bh[1][0], bl[1][0]); split_pair(v[2].y, v[3].y, bh[1][1], bl[1][1]);
      split_pair(v[0].z, v[1].z, bh[2][0], bl[2][0]); split_pair(v[2].z, v[3].z, bh[2][1], bl[2][1]);
      split_pair(v[0].w, v[1].w, bh[3][0], bl[3][0]); split_pair(v[2].w, v[3].w, bh[3][1], bl[3][1]);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        unsigned ah[4], al[4];
        sm_ldsm_x4(ah, &qh[16 * m + (l & 15)][16 * ks + (l >> 4) * 8]);
        sm_ldsm_x4(al, &ql[16 * m + (l & 15)][16 * ks + (l >> 4) * 8]);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) sm_mma(acc[m][nt], ah, bh[nt][0], bh[nt][1]);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) sm_mma(acc[m][nt], al, bh[nt][0], bh[nt][1]);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) sm_mma(acc[m][nt], ah, bl[nt][0], bl[nt][1]);
      }
    }
    // relu per head and the sum over the four heads of a row: lanes g, g ^ 1, g ^ 2, g ^ 3 hold the heads of the span rows
    // 4 m + g / 4 (accumulator row g) and + 2 (row g + 8), columns 2 tq and 2 tq + 1.  Every exchange gives away half of what a
    // lane holds, so that in the end lane g has the four blocks of column 2 tq + (g & 1) of row 4 m + 2 (g >> 1 & 1) + g / 4.
    const bool odd = g & 1, lower = g & 2;
    const int blk = (first + (s0 >> 3)) * 32 + 8 * tq + (odd ? 4 : 0);
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      float sc[4];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        float half[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const float c0 = fmaxf(acc[m][nt][2 * k], 0.f), c1 = fmaxf(acc[m][nt][2 * k + 1], 0.f);
          half[k] = (odd ? c1 : c0) + __shfl_xor_sync(0xffffffffu, odd ? c0 : c1, 4);
        }
        sc[nt] = ((lower ? half[1] : half[0]) + __shfl_xor_sync(0xffffffffu, lower ? half[0] : half[1], 8)) * kInvSqrt128;
      }
      const int r = 4 * m + (lower ? 2 : 0) + (g >> 2);
      const int nb = (a.pos0 + r + 1) / 4;
      if (r >= a.R || nb <= CR_SEL_BLOCKS) continue;
      float* dst = a.scores + (size_t)r * a.sstride + blk;
      if (blk + 4 <= nb && ((uintptr_t)dst & 15) == 0) {
        *reinterpret_cast<float4*>(dst) = make_float4(sc[0], sc[1], sc[2], sc[3]);
      } else {
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
          if (blk + nt < nb) dst[nt] = sc[nt];
      }
    }
  }
}

// Spans of 3..16 rows, every block of every row.  Three CTAs of four warps fit an SM; the tiles are dealt in one wave of them.  (Dealt over
// all warps, whatever the spans' last CTAs held, 16 spans of 111 tiles came to 448 CTAs for 444 places: 11.2 us for 4 rows, 9.8
// now; 8 of 1,110 tiles 38.0 and 30.5, of 9 rows 50.8 and 44.6.)  13 to 16 rows, 168 registers a thread with 24 bytes spilled: 8 sessions at 131,072
// positions 50.5 us, 66 to 68 in the form of half a tile a step with four CTAs to an SM.
cr_status qsa_score_mma_launch(const QsaParams& P, int tiles, int Rmax, int n, bool wide, cudaStream_t stream) {
  const int per_warp = score_tiles_per_warp(tiles, n, sm_count());
  const dim3 grid((tiles + 4 * per_warp - 1) / (4 * per_warp), 1, n);
  const int mt = (Rmax + 3) / 4;
  auto pick = [&](auto w) {
    constexpr bool W = decltype(w)::value;
    return mt <= 1 ? qsa_score_mma_kernel<1, W> : mt == 2 ? qsa_score_mma_kernel<2, W> : mt == 3 ? qsa_score_mma_kernel<3, W> : qsa_score_mma_kernel<4, W>;
  };
  CR_CUDA(launch_pdl(wide ? pick(std::true_type{}) : pick(std::false_type{}), grid, dim3(128), 0, stream, P, per_warp));
  CR_LAUNCH_CHECK("qsa_score_mma_kernel");
  return CR_OK;
}

}  // namespace cr

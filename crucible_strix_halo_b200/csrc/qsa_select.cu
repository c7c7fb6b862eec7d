// QSA block selection for sm_100a: indexer scores over the pooled keys.
//
// Scores (QsaScoreKernel / QsaScoreRowsKernel, engine/layers/qsa_long.h:9-108): HBM-bound scan of the tiled
// fp32 pool [b/32][128][32].  One warp owns one 16 KB tile: lane = block, every load of the warp is one full
// 128-byte line, and a group of up to RT rows is scored from one read of the tile.
//
// The exact top-512 over these scores is in qsa_topk.cu.
#include <climits>
#include "qsa.cuh"

namespace cr {

// ---- scores --------------------------------------------------------------------------------------------
// grid (ceil(tiles/8), row groups, spans), 256 threads; blockIdx.y = group of RT consecutive rows.
template <int RT, bool RANGED>
__global__ void __launch_bounds__(256) qsa_score_kernel(const __grid_constant__ QsaParams P) {
  const cr_qsa_args& a = P.span[blockIdx.z];
  const int rg0 = blockIdx.y * RT;
  if (rg0 >= a.R) return;
  const int nr = min(RT, a.R - rg0);
  const int nb_all = (a.pos0 + rg0 + nr) / 4;       // blocks complete for the last row of the group
  if (nb_all <= CR_SEL_BLOCKS) return;
  const int nb_hi = RANGED ? min(nb_all, P.b_hi) : nb_all;   // the scored range ends here
  const int t = threadIdx.x, w = t >> 5, l = t & 31;
  __shared__ float4 iqs[128][RT];                    // [dim][row] = the 4 indexer heads
  for (int i = t; i < 128 * RT; i += 256) {
    const int d = i / RT, r = i % RT;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < nr) {
      const float* iq = a.idx + (size_t)(rg0 + r) * 640;
      v = make_float4(iq[d], iq[128 + d], iq[256 + d], iq[384 + d]);
    }
    iqs[d][r] = v;
  }
  __syncthreads();
  const int tile = (RANGED ? P.b_lo / 32 : 0) + blockIdx.x * 8 + w;
  if (tile * 32 >= nb_hi) return;
  const int b = tile * 32 + l;
  const float* pt = a.c.ik_pool + (size_t)tile * 4096 + l;
  float acc[RT][4];
#pragma unroll
  for (int r = 0; r < RT; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
#pragma unroll 4
  for (int d0 = 0; d0 < 128; d0 += 16) {
    float key[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) key[j] = __ldg(pt + (d0 + j) * 32);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        const float4 q = iqs[d0 + j][r];
        acc[r][0] = fmaf(q.x, key[j], acc[r][0]);
        acc[r][1] = fmaf(q.y, key[j], acc[r][1]);
        acc[r][2] = fmaf(q.z, key[j], acc[r][2]);
        acc[r][3] = fmaf(q.w, key[j], acc[r][3]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    if (r >= nr) break;
    const int nb = (a.pos0 + rg0 + r + 1) / 4;
    if (nb <= CR_SEL_BLOCKS || b >= nb) continue;
    if constexpr (RANGED) { if (b < P.b_lo || b >= P.b_hi) continue; }
    float s = fmaxf(acc[r][0], 0.f);
    s += fmaxf(acc[r][1], 0.f);
    s += fmaxf(acc[r][2], 0.f);
    s += fmaxf(acc[r][3], 0.f);
    a.scores[(size_t)(rg0 + r) * a.sstride + b] = s * kInvSqrt128;
  }
}

// Same scores for one or two rows with 128-bit loads: lane l reads blocks 4(l%8)..+3 of dims l/8, l/8+4, ...,
// so a warp load covers four 128-byte lines and the tile costs 32 load instructions per lane instead of 128.
// The four lanes that share a block group add their partial dots with two shuffles.
// The pool passes through L2 as the first thing to be evicted: four sessions of 262,144 positions (134 MB, more than L2) had pushed
// out the states, the rows and the code of the kernels around the scan: a step 75.4 -> 66.1 us, of which 4 in the attention.
// Half a tile is asked for before the queries are staged and stays in flight: 60.0 -> 58.6 us for passes back to back.  (Asking the
// tiles into L2 before the wait for the kernel ahead was slower: the prefetches come in with the ordinary policy.)
// RANGED: only the blocks [P.b_lo, P.b_hi) are scored (a rank's own blocks).  A separate instantiation: with the range
// tests in it the whole-row kernel measured 40 us instead of 29 for four 262,144-token rows.
// AHEAD: with half a tile in flight from the start two CTAs of 101 or 123 registers a thread fit an SM; without it four of two rows, a
// quarter of a tile at a time.  score4_ahead() has the line.
template <int RT, bool RANGED, bool AHEAD>
__global__ void __launch_bounds__(256, AHEAD ? 0 : 4) qsa_score4_kernel(const __grid_constant__ QsaParams P) {
  pdl_release();
  const cr_qsa_args& a = P.span[blockIdx.z];
  touch_params(a);
  pdl_wait();
  const int rg0 = blockIdx.y * RT;
  if (rg0 >= a.R) return;
  const int nr = min(RT, a.R - rg0);
  const int nb_all = (a.pos0 + rg0 + nr) / 4;
  if (nb_all <= CR_SEL_BLOCKS) return;
  const int nb_hi = RANGED ? min(nb_all, P.b_hi) : nb_all;
  const int t = threadIdx.x, w = t >> 5, l = t & 31;
  __shared__ float4 iqs[128][RT];
  const int tile = (RANGED ? P.b_lo / 32 : 0) + blockIdx.x * 8 + w;
  const bool live = tile * 32 < nb_hi;
  const int bq = (l & 7) * 4, dl = l >> 3;
  const float* pt = a.c.ik_pool + (size_t)tile * 4096 + dl * 32 + bq;
  const uint64_t policy = evict_first_policy();
  float4 key[AHEAD ? 2 : 1][8];               // a quarter of the tile each
  auto fetch = [&](float4 (&k)[8], int it0) {
#pragma unroll
    for (int j = 0; j < 8; ++j) k[j] = load_stream4(pt + (it0 + j) * 128, policy);
  };
  if constexpr (AHEAD) {
    if (live) { fetch(key[0], 0); fetch(key[1], 8); }             // in flight while the queries are staged
  }
  for (int i = t; i < 128 * RT; i += 256) {
    const int d = i / RT, r = i % RT;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < nr) {
      const float* iq = a.idx + (size_t)(rg0 + r) * 640;
      v = make_float4(iq[d], iq[128 + d], iq[256 + d], iq[384 + d]);
    }
    iqs[d][r] = v;
  }
  __syncthreads();
  if (!live) return;
  float acc[RT][4][4];                        // [row][block][head]
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[r][b][0] = acc[r][b][1] = acc[r][b][2] = acc[r][b][3] = 0.f;
#pragma unroll
  for (int it0 = 0; it0 < 32; it0 += 8) {
    float4 (&k)[8] = key[AHEAD ? (it0 >> 3) & 1 : 0];
    if constexpr (!AHEAD) fetch(k, it0);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float kb[4] = {k[j].x, k[j].y, k[j].z, k[j].w};
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        const float4 q = iqs[(it0 + j) * 4 + dl][r];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          acc[r][b][0] = fmaf(q.x, kb[b], acc[r][b][0]);
          acc[r][b][1] = fmaf(q.y, kb[b], acc[r][b][1]);
          acc[r][b][2] = fmaf(q.z, kb[b], acc[r][b][2]);
          acc[r][b][3] = fmaf(q.w, kb[b], acc[r][b][3]);
        }
      }
    }
    if constexpr (AHEAD) {
      if (it0 + 16 < 32) fetch(k, it0 + 16);
    }
  }
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        acc[r][b][h] += __shfl_xor_sync(0xffffffffu, acc[r][b][h], 8);
        acc[r][b][h] += __shfl_xor_sync(0xffffffffu, acc[r][b][h], 16);
      }
  if (dl != 0) return;
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    if (r >= nr) break;
    const int nb = (a.pos0 + rg0 + r + 1) / 4;
    if (nb <= CR_SEL_BLOCKS) continue;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int blk = tile * 32 + bq + b;
      if (blk >= nb) continue;
      if constexpr (RANGED) { if (blk < P.b_lo || blk >= P.b_hi) continue; }
      float s = fmaxf(acc[r][b][0], 0.f);
      s += fmaxf(acc[r][b][1], 0.f);
      s += fmaxf(acc[r][b][2], 0.f);
      s += fmaxf(acc[r][b][3], 0.f);
      a.scores[(size_t)(rg0 + r) * a.sstride + blk] = s * kInvSqrt128;
    }
  }
}

template <int RT>
static cr_status score_launch_t(const QsaParams& P, int tiles, int Rmax, int n, bool ranged, cudaStream_t stream) {
  const dim3 grid((tiles + 7) / 8, (Rmax + RT - 1) / RT, n);
  if (ranged) qsa_score_kernel<RT, true><<<grid, 256, 0, stream>>>(P);
  else qsa_score_kernel<RT, false><<<grid, 256, 0, stream>>>(P);
  CR_LAUNCH_CHECK("qsa_score_kernel");
  return CR_OK;
}

// Whether a launch of `ctas` CTAs of qsa_score4_kernel has the loads of half a tile in flight from the start: all but whole rows in pairs
// where that form's CTAs need a second wave and those of the other do not.  Two rows each, us in the one form | the other: pool in L2, 4 sessions
// of 20,000 blocks 10.9 | 9.3, 8 of 14,000 11.6 | 9.8, 4 of 32,768 12.1 | 11.8; from HBM 13.5 | 11.7, 14.7 | 13.6, 15.6 | 15.2; on either side of
// the range 4 of 8,001 5.2 | 5.5, 8 of 32,768 24.9 | 26.1.  One row: L2 7.6 | 6.4 and 9.2 | 7.9 for 4 sessions of 20,000 and 32,768 blocks, but HBM
// 10.3 | 10.5 and 13.5 | 14.3, where the pools of a model with several layers are.  A range of 131,072 blocks: 12.3 | 12.0.
static bool score4_ahead(int rows, bool ranged, long long ctas) { return rows == 1 || ranged || ctas <= 2 * sm_count() || ctas > 4 * sm_count(); }

cr_status qsa_score_launch(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, cudaStream_t stream, int b_lo, int b_hi) {
  use_stream(stream);
  for (int s0 = 0; s0 < n_spans; s0 += kMaxSpans) {
    const int n = n_spans - s0 < kMaxSpans ? n_spans - s0 : kMaxSpans;
    QsaParams P;
    qsa_fill_params(P, g, spans + s0, n);
    P.b_lo = b_lo; P.b_hi = b_hi;
    const bool ranged = b_lo > 0 || b_hi < INT_MAX;
    const int Rmax = qsa_max_rows(spans + s0, n);
    int nb_max = 0;
    bool wide = true;                               // every pool at a 16-byte boundary: loads of four blocks, else of one
    for (int s = 0; s < n; ++s) {
      nb_max = max(nb_max, (spans[s0 + s].pos0 + spans[s0 + s].R) / 4);
      wide &= ((uintptr_t)spans[s0 + s].c.ik_pool & 15) == 0;
    }
    if (nb_max <= CR_SEL_BLOCKS) continue;
    const int hi = nb_max < b_hi ? nb_max : b_hi;
    if (hi <= b_lo) continue;                       // the range holds no complete block of these rows
    const int tiles = (hi + 31) / 32 - b_lo / 32;   // 32-block pool tiles that overlap the scored range
    cr_status st;
    if (Rmax <= 2 && wide) {
      const dim3 grid((tiles + 7) / 8, 1, n);
      const bool ahead = score4_ahead(Rmax, ranged, (long long)grid.x * n);
      auto kernel = Rmax == 1 ? (ranged ? qsa_score4_kernel<1, true, true> : qsa_score4_kernel<1, false, true>)
                    : ranged  ? qsa_score4_kernel<2, true, true>
                              : (ahead ? qsa_score4_kernel<2, false, true> : qsa_score4_kernel<2, false, false>);
      CR_CUDA(launch_pdl(kernel, grid, dim3(256), 0, stream, P));
      CR_LAUNCH_CHECK("qsa_score_kernel");
      st = CR_OK;
    }
    else if (Rmax > 2 && Rmax <= 16 && !ranged && !options().qsa_score_simt) st = qsa_score_mma_launch(P, tiles, Rmax, n, wide, stream);   // verify spans
    else if (Rmax >= 8 && !options().qsa_score_simt) st = qsa_score_tc_launch(P, n, stream);   // prefill parts (and a rank's range of a span)
    else if (Rmax <= 4) st = score_launch_t<4>(P, tiles, Rmax, n, ranged, stream);
    else st = score_launch_t<8>(P, tiles, Rmax, n, ranged, stream);
    if (st) return st;
  }
  return CR_OK;
}

cr_status qsa_select_launch(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, cudaStream_t stream, bool dense_marked) {
  if (cr_status s = qsa_score_launch(g, spans, n_spans, stream)) return s;
  return qsa_topk_launch(g, spans, n_spans, stream, dense_marked);
}

}  // namespace cr

extern "C" size_t cr_qsa_select_scratch_bytes(const cr_geometry*, int) { return 0; }

extern "C" cr_status cr_qsa_select(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, void*, size_t, void* stream) {
  using namespace cr;
  if (cr_status s = qsa_validate(g, spans, n_spans, CR_MAX_PREFILL_ROWS, "cr_qsa_select")) return s;
  return qsa_select_launch(g, spans, n_spans, (cudaStream_t)stream);
}

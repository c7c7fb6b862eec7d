// qsa_score_tc_kernel: indexer scores of a prefill part on tcgen05 tensor cores (kind::f16) (QsaPrefillSgprScoreKernel,
// engine/layers/kernels/prefill_qsa_score_sgpr.h:19-81, computes the same scores with fp32 FMAs).
//
//   score[r][b] = (sum_{h<4} max(iq[r][h] . pool[b], 0)) / sqrt(128)        for b < (pos0 + r + 1) / 4
//
// is four GEMMs of shape [blocks x 128] x [128 x rows] with a ReLU between them and their sum.  A CTA pair (tcgen05
// cta_group::2) owns 64 rows and a run of pool tiles of 256 blocks, 128 in each CTA: M = 256 blocks (the pool tile is the A
// operand), N = 256 = 4 heads x 64 rows, K = 128.  Each CTA keeps half of the query panel (two heads, 64 KB) in shared memory
// as its half of the B operand, which leaves room for two pool tiles: one is staged while the other is multiplied.  The heads
// are the four 64-column quarters of a TMEM accumulator, two accumulators used in turn, so the epilogue of a tile (ReLU, sum
// over heads, scale, store) runs beside the next ones too.  The visits (row tile, pool tile) of a span are dealt to the pairs
// in equal runs; a pair reloads its panel where its run enters the next row tile.
// Precision: both operands are split into an fp16 head and an fp16 remainder (22 mantissa bits together; the values are
// normalised rows, well inside the fp16 range) and three products are accumulated in fp32 (head x head, head x remainder,
// remainder x head); the error of a score stays below 1e-5 (measured 9e-6 against fp64 scores of the same operands; 4e-6 for
// the fp32 FMA kernel), far inside the 1e-3 gap within which selections may differ.  The pool is stored [dim][32 blocks] per
// 32-block tile, i.e. transposed for a K-major operand: eight staging warps read it with coalesced loads, split it and write
// 16-byte K-major units.  Every wait is bounded and raises a status word.
// Bound: the tensor pipe, 24 MMAs of 129 cycles per 128 blocks and 64 rows.  With the whole panel in one CTA there was room for
// one pool tile, so that staging and multiplying took turns, and four epilogue warps of 64 rows a lane took 8,400 cycles a tile
// (eight of 32 rows: 2,600): 2,048 rows at 260,096 453 us, 345 us now; at 30,720 76 -> 60 us; 117 rows at 9,003 13.5 -> 12 us.
#include <algorithm>
#include <climits>
#include <cooperative_groups.h>
#include "qsa.cuh"
#include "umma.cuh"

namespace cg = cooperative_groups;

namespace cr {

CR_DEFINE_STATUS_WORD(qsa_score)

constexpr int kScRows = 64;                 // query rows per CTA (N)
constexpr int kScBlocks = 128;              // pool blocks per tile of a CTA (half of M)
constexpr int kScStage = 8, kScIssuer = 16;  // first staging warp (after 8 epilogue warps), issuer warp (after 8 staging warps)
constexpr int kScThreads = 32 * (kScIssuer + 1);
constexpr int kQopBytes = 2 * 16 * 2 * kScRows * 16;      // [hi/lo][dim / 8][two heads][row][8 fp16]: 128 of the N = 256 columns
constexpr int kPopBytes = 2 * 16 * kScBlocks * 16;        // [hi/lo][dim / 8][block][8 fp16]; two of them
constexpr size_t kScoreSmem = kQopBytes + 2 * kPopBytes + 128;

__host__ __device__ constexpr uint32_t idesc_f16(int M, int N) { return umma::idesc_f16(M, N, false, false); }
// eight fp32 values -> fp16 heads and fp16 remainders, each packed into 16 bytes
__device__ __forceinline__ void split8(const float (&x)[8], uint4& hi, uint4& lo) {
  unsigned h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half2 a = __floats2half2_rn(x[2 * i], x[2 * i + 1]);
    const float2 b = __half22float2(a);
    const __half2 c = __floats2half2_rn(x[2 * i] - b.x, x[2 * i + 1] - b.y);
    h[i] = *reinterpret_cast<const unsigned*>(&a);
    l[i] = *reinterpret_cast<const unsigned*>(&c);
  }
  hi = make_uint4(h[0], h[1], h[2], h[3]);
  lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// Pool tiles (of 256 blocks) that row tile rt of a span scores: [lo, lo + count).
__host__ __device__ __forceinline__ int score_tiles(int pos0, int R, int rt, int b_lo, int b_hi, int& lo) {
  const int end = R < (rt + 1) * kScRows ? R : (rt + 1) * kScRows, nb_all = (pos0 + end) / 4;   // blocks visible to the tile's last row
  lo = b_lo / (2 * kScBlocks);
  if (nb_all <= CR_SEL_BLOCKS) return 0;                  // dense rows
  const int hi = ((nb_all < b_hi ? nb_all : b_hi) + 2 * kScBlocks - 1) / (2 * kScBlocks);
  return hi > lo ? hi - lo : 0;
}

// grid (pairs x 2, 1, spans), clusters of 2.  RANGED: the scored range [b_lo, b_hi) of a rank.
template <bool RANGED>
__global__ void __launch_bounds__(kScThreads, 1) qsa_score_tc_kernel(const __grid_constant__ QsaParams P) {
  extern __shared__ __align__(128) unsigned char sm[];
  unsigned char* Qop = sm;
  unsigned char* Pops = sm + kQopBytes;
  __shared__ __align__(8) uint64_t bars[6];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int dead;
  uint64_t *popFull = &bars[0], *mmaDone = &bars[2], *accFree = &bars[4];    // one per buffer; popFull and accFree: the leader's
  const cr_qsa_args& a = P.span[blockIdx.z];
  const int b_lo = RANGED ? P.b_lo : 0, b_hi = RANGED ? P.b_hi : INT_MAX;
  const int t = threadIdx.x, w = t >> 5, l = t & 31;
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t rank = cluster.block_rank();             // 0 leads
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1, row_tiles = (a.R + kScRows - 1) / kScRows;
  int visits = 0;
  for (int rt = 0; rt < row_tiles; ++rt) { int lo; visits += score_tiles(a.pos0, a.R, rt, b_lo, b_hi, lo); }
  const int v0 = (int)((long long)visits * pair / pairs), v1 = (int)((long long)visits * (pair + 1) / pairs);
  if (v0 >= v1) return;                                   // both CTAs of the pair

  if (t == 0) {
    for (int i = 0; i < 2; ++i) {
      umma::mbar_init(&popFull[i], 16);                   // one arrival per staging warp of both CTAs
      umma::mbar_init(&mmaDone[i], 1);
      umma::mbar_init(&accFree[i], 16);                   // one arrival per epilogue warp of both CTAs
    }
    umma::mbar_fence_init();
    dead = 0;
  }
  if (w == kScIssuer) umma::pair_tmem_alloc(&tmem_slot, 512);
  bool gave_up = false;
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if (gave_up) return;
    if (!umma::mbar_wait_timed(bar, parity, &dead)) { gave_up = true; dead = 1; g_qsa_score_status = 1; }
  };

  int n0 = 0;                                             // visits of this pair before the current row tile
  int first = 0;                                          // first visit of row tile rt
  for (int rt = 0; rt < row_tiles && first < v1; ++rt) {
    int lo;
    const int count = score_tiles(a.pos0, a.R, rt, b_lo, b_hi, lo);
    const int t0 = lo + max(v0 - first, 0), t1 = lo + min(v1 - first, count);
    first += count;
    if (t0 >= t1) continue;
    const int r0 = rt * kScRows, rows = min(kScRows, a.R - r0), nb_hi = min((a.pos0 + r0 + rows) / 4, b_hi);
    // query panel: rows r0 .. r0+63 of two indexer heads, split and stored K-major
    for (int i = t; i < 2 * 16 * kScRows; i += kScThreads) {
      const int row = i % kScRows, dc = (i / kScRows) % 16, h = i / (kScRows * 16);
      float x[8];
      if (row < rows) {
        const float4* src = reinterpret_cast<const float4*>(a.idx + (size_t)(r0 + row) * 640 + (2 * rank + h) * 128 + dc * 8);
        const float4 u = src[0], v = src[1];
        x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w; x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = 0.f;
      }
      uint4 hi, lo16;
      split8(x, hi, lo16);
      *reinterpret_cast<uint4*>(Qop + ((size_t)(dc * 2 + h) * kScRows + row) * 16) = hi;
      *reinterpret_cast<uint4*>(Qop + kQopBytes / 2 + ((size_t)(dc * 2 + h) * kScRows + row) * 16) = lo16;
    }
    umma::fence_async_smem();
    umma::fence_before_sync();
    cluster.sync();                                       // both panels are there (and, the first time, the barriers)
    umma::fence_after_sync();
    const uint32_t tm = tmem_slot;

    if (w == kScIssuer) {
      // ---------------------------------------------------------------- issuer (of the leader)
      if (l == 0 && rank == 0) {
        constexpr uint32_t idesc = idesc_f16(2 * kScBlocks, 4 * kScRows);
        const uint64_t dQh = umma::smem_desc(Qop, 2 * kScRows * 16, 128), dQl = umma::smem_desc(Qop + kQopBytes / 2, 2 * kScRows * 16, 128);
        for (int i = n0; i < n0 + t1 - t0; ++i) {
          const int buf = i & 1;
          const unsigned char* Pop = Pops + buf * kPopBytes;
          const uint64_t dPh = umma::smem_desc(Pop, kScBlocks * 16, 128), dPl = umma::smem_desc(Pop + kPopBytes / 2, kScBlocks * 16, 128);
          wait(&popFull[buf], (i >> 1) & 1);
          if (i >= 2) wait(&accFree[buf], ((i >> 1) - 1) & 1);
          if (gave_up || dead) break;                      // no more tensor-core work once any wait has run out
          asm volatile("fence.acq_rel.cluster;\n" ::: "memory");   // the other CTA's tile
          umma::fence_after_sync();
          const uint32_t d = tm + buf * 256;
          // a step of 16 along K is two 16-byte planes of 128 units, in the pool tile and in the query panel
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) umma::pair_mma(d, dPh + (uint64_t)(ks * 256), dQh + (uint64_t)(ks * 256), idesc, ks > 0);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) umma::pair_mma(d, dPh + (uint64_t)(ks * 256), dQl + (uint64_t)(ks * 256), idesc, 1u);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) umma::pair_mma(d, dPl + (uint64_t)(ks * 256), dQh + (uint64_t)(ks * 256), idesc, 1u);
          umma::pair_commit(&mmaDone[buf]);
        }
      }
    } else if (w >= kScStage) {
      // ---------------------------------------------------------------- staging warps: pool tile -> K-major fp16 head + remainder
      const int sw = w - kScStage, sb = sw & 3, dc0 = (sw >> 2) * 8;      // 32-block sub-tile, first of its 8 dim chunks
      const int blk = sb * 32 + l;
      for (int i = n0; i < n0 + t1 - t0; ++i) {
        const int tile = 2 * (t0 + i - n0) + rank;
        unsigned char* Pop = Pops + (i & 1) * kPopBytes;
        const bool live = tile * kScBlocks + sb * 32 < nb_hi;       // the pool is allocated in whole 32-block tiles
        const float* src = a.c.ik_pool + ((size_t)tile * 4 + sb) * 4096 + l;
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          float x[4][8];
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int j = 0; j < 8; ++j) x[c][j] = live ? __ldg(src + ((dc0 + 4 * part + c) * 8 + j) * 32) : 0.f;
          if (part == 0 && i >= 2) {                                // the MMAs that read this buffer are done
            if (l == 0) wait(&mmaDone[i & 1], ((i >> 1) - 1) & 1);
            __syncwarp();
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint4 hi, lo16;
            split8(x[c], hi, lo16);
            *reinterpret_cast<uint4*>(Pop + ((size_t)(dc0 + 4 * part + c) * kScBlocks + blk) * 16) = hi;
            *reinterpret_cast<uint4*>(Pop + kPopBytes / 2 + ((size_t)(dc0 + 4 * part + c) * kScBlocks + blk) * 16) = lo16;
          }
        }
        umma::fence_async_smem();
        __syncwarp();
        if (l == 0) umma::pair_arrive(umma::cluster_addr(&popFull[i & 1], 0));
      }
    } else {
      // ---------------------------------------------------------------- epilogue warps: lane = TMEM lane = block of the tile,
      // warps 0-3 the first 32 rows, 4-7 the last
      const int row0 = (w >> 2) * 32;
      for (int i = n0; i < n0 + t1 - t0; ++i) {
        const int buf = i & 1, b = (2 * (t0 + i - n0) + (int)rank) * kScBlocks + (t & 127);
        if (l == 0) wait(&mmaDone[buf], (i >> 1) & 1);
        __syncwarp();
        umma::fence_after_sync();
        float s[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) s[c] = 0.f;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          float p[32];
          umma::tmem_ld32(umma::tmem_addr(tm, w, buf * 256 + h * 64 + row0), p);
#pragma unroll
          for (int c = 0; c < 32; ++c) s[c] += fmaxf(p[c], 0.f);
        }
        umma::fence_before_sync();
        __syncwarp();
        if (l == 0) umma::pair_arrive_relaxed(umma::cluster_addr(&accFree[buf], 0));
        if (b < nb_hi && (!RANGED || b >= b_lo)) {
          float* dst = a.scores + (size_t)(r0 + row0) * a.sstride + b;
#pragma unroll
          for (int c = 0; c < 32; ++c, dst += a.sstride)
            if (row0 + c < rows) *dst = s[c] * kInvSqrt128;
        }
      }
    }
    n0 += t1 - t0;
    __syncwarp();
    // Every MMA of this row tile has completed (the epilogue warps of both CTAs waited for them): the panel may change.
    umma::fence_before_sync();
    cluster.sync();
    umma::fence_after_sync();
  }
  if (w == kScIssuer) umma::pair_tmem_dealloc(tmem_slot, 512);
}

cr_status qsa_score_tc_launch(const QsaParams& P, int n, cudaStream_t stream) {
  static PerDeviceOnce configured;
  if (cr_status st = once_per_device(configured, [] {
        CR_CUDA(cudaFuncSetAttribute(qsa_score_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScoreSmem));
        CR_CUDA(cudaFuncSetAttribute(qsa_score_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScoreSmem));
        return CR_OK;
      })) return st;
  // One CTA per SM (192 KB of shared memory, all of TMEM), one wave; no more pairs than the longest span has visits.
  const bool ranged = P.b_lo > 0 || P.b_hi < INT_MAX;
  long long most = 0;
  for (int i = 0; i < n; ++i) {
    long long visits = 0;
    for (int rt = 0; rt * kScRows < P.span[i].R; ++rt) { int lo; visits += score_tiles(P.span[i].pos0, P.span[i].R, rt, ranged ? P.b_lo : 0, ranged ? P.b_hi : INT_MAX, lo); }
    if (visits > most) most = visits;
  }
  if (most == 0) return CR_OK;
  int pairs = sm_count() / 2 / n;
  pairs = (int)std::min<long long>(pairs < 1 ? 1 : pairs, most);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs, 1, n); cfg.blockDim = dim3(kScThreads); cfg.dynamicSmemBytes = kScoreSmem; cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  CR_CUDA(cudaLaunchKernelEx(&cfg, ranged ? qsa_score_tc_kernel<true> : qsa_score_tc_kernel<false>, P));
  CR_LAUNCH_CHECK("qsa_score_tc_kernel");
  return CR_OK;
}

}  // namespace cr

// Projection GEMM either side of the attention core for sm_100a: Y[R][N] = X[R][K] W[N][K]^T with bf16 operands and
// fp32 accumulation, the columns of Y scattered straight into the buffers the core reads (qkv / z / gate logits of a
// GDN layer, q / k / v / idx of a QSA layer) or, on the way out, the hidden rows.  The role of the input and output
// GEMM groups of a prefill layer (PrefillLayer::input / ::output, engine/runtime/prefill_engine.inc:261-270, :362)
// for plain bf16 weights; the reference's EXL3 trellis decoding is not part of this path.
//
// proj_gemm_pair_kernel (many rows): CTA pairs on 256 x 256 tiles.  A CTA's shared memory moves 128 bytes a cycle; a
// 128 x 256 tile of one CTA reads 12 KB and takes in 12 KB per K step of 16, 188 cycles of it against 129 cycles of tensor
// pipe, and that set the pace.  tcgen05.mma.cta_group::2 multiplies 256 rows (128 of X in each CTA) by 256 columns
// (128 of W in each CTA): 8 + 8 KB per step, the pipe's own 128 cycles.  Persistent, six warps per CTA:
//   warp 0    producer: its own halves of the X and W tiles (128 x 64 boxes) into a six-stage ring of 128-byte-swizzled
//             tiles; the bytes of both CTAs complete on the leader's barrier;
//   warp 1    issuer (leader only): four MMAs per stage into one of two 256-column accumulators; commits arrive in both CTAs;
//   warps 2-5 epilogue: tcgen05.ld of the warp's 32 lanes, conversion, row stores into the output that owns the 32-column
//             chunk; the other accumulator is filled meanwhile.
// 32,768 x 2,048 x 12,352: 1,283 us on single CTAs, 1,132 us now (1.47 PFLOP/s); 16,384 x 2,048 x 9,856: 508 -> 438 us.
//
// proj_gemm_split_kernel<TN> (few rows): a 128 x TN tile and a share of K per CTA.  Short calls have fewer tiles than SMs
// and are bound by how fast W arrives: the split of K over a cluster of up to eight CTAs lets every SM pull its part, and
// the partial tiles are summed through distributed shared memory, a slice of rows per CTA, with whole rows stored.  W cold
// in L2, against 128 x 128 or 128 x 256 tiles without a split: 333 x 4,096 x 2,048 27.9 -> 14.7 us, 333 x 6,144 x 2,560
// 41.6 -> 19.7 us, 64 x 4,096 x 2,048 25.4 -> 9.6 us, 1 or 64 x 2,048 x 12,352 18.4 -> 15.3 us, 333 x 2,048 x 12,352
// 21.6 -> 21.2 us (147 tiles of 128 x 256 either way: one wave, shared-memory bound).
//
// Tiles are walked in bands of column tiles, so that a wave of CTAs shares W and X tiles through L2.  Rows and columns past
// the matrix are zero-filled by the copy engine and masked in the epilogue.  Every wait is bounded; a wait that gives up
// raises bit 4 of the device status word.
#include <cooperative_groups.h>
#include "common.cuh"
#include "tma.cuh"
#include "umma.cuh"

namespace cg = cooperative_groups;

namespace cr {

CR_DEFINE_STATUS_WORD(proj_gemm)

constexpr int kGM = 128, kGK = 64;
constexpr int kGThreads = 192;
constexpr int kMaxOuts = 6;
constexpr int kTileBytes = kGM * kGK * 2;                       // 128 rows x 64 channels of X or W

struct ProjParams {
  int R, K, N, n_outs;
  void* ptr[kMaxOuts];
  int col0[kMaxOuts], cols[kMaxOuts], ld[kMaxOuts], f32[kMaxOuts];
};

__device__ __forceinline__ void load_box_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
                   umma::smem_u32(dst)),
               "l"(map), "r"(c0), "r"(c1), "r"(umma::smem_u32(bar))
               : "memory");
}
// Instruction descriptor for kind::f16 with bf16 operands (format 1), fp32 accumulation, both operands K-major.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// ---- CTA pairs: the cta_group::2 forms --------------------------------------------------------------------------
// A box into this CTA's shared memory whose bytes complete on a barrier of either CTA of the pair.
__device__ __forceinline__ void pair_load_box_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
                   umma::smem_u32(dst)),
               "l"(map), "r"(c0), "r"(c1), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) { asm volatile("prefetch.tensormap [%0];\n" ::"l"(map) : "memory"); }

// Columns col .. col + 31 of one row to the output that owns them.
__device__ __forceinline__ void store_chunk(const ProjParams& P, int row, int col, const float (&v)[32]) {
  int o = 0;
  while (o < P.n_outs - 1 && col >= P.col0[o] + P.cols[o]) ++o;       // outputs are ordered by column; chunks do not straddle them
  const size_t at = (size_t)row * P.ld[o] + (col - P.col0[o]);
  if (P.f32[o]) {
    float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(P.ptr[o]) + at);
#pragma unroll
    for (int k = 0; k < 8; ++k) dst[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
  } else {
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(P.ptr[o]) + at);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      unsigned pk[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __nv_bfloat162 b2 = __floats2bfloat162_rn(v[8 * k + 2 * j], v[8 * k + 2 * j + 1]);
        pk[j] = *reinterpret_cast<const unsigned*>(&b2);
      }
      dst[k] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
    }
  }
}
// Four columns of one row.
__device__ __forceinline__ void store_quad(const ProjParams& P, int row, int col, const float4 v) {
  int o = 0;
  while (o < P.n_outs - 1 && col >= P.col0[o] + P.cols[o]) ++o;
  const size_t at = (size_t)row * P.ld[o] + (col - P.col0[o]);
  if (P.f32[o]) *reinterpret_cast<float4*>(reinterpret_cast<float*>(P.ptr[o]) + at) = v;
  else {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(P.ptr[o]) + at) =
        make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
  }
}

// ---- CTA pairs on 256 x 256 tiles ----------------------------------------------------------------------------------
constexpr int kPStages = 6, kPStageBytes = 2 * kTileBytes, kPBand = 16;
constexpr size_t kPairSmem = (size_t)kPStages * kPStageBytes + (2 * kPStages + 4) * 8 + 16;

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGThreads, 1)
proj_gemm_pair_kernel(const __grid_constant__ ProjParams P, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap) {
  extern __shared__ __align__(1024) unsigned char sm[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + kPStages * kPStageBytes);
  uint64_t *full = bars, *empty = bars + kPStages, *accFull = bars + 2 * kPStages, *accEmpty = bars + 2 * kPStages + 2;
  uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 2 * kPStages + 4);
  volatile int& dead = *reinterpret_cast<volatile int*>(&tmem_slot + 1);
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t rank = cluster.block_rank();                          // 0 leads
  const int t = threadIdx.x, w = t >> 5, l = t & 31;
  const int mt = (P.R + 255) / 256, nt = (P.N + 255) / 256, kb_n = P.K / kGK, tiles = mt * nt;
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  auto tile_at = [&](int i, int& m0, int& n0) {
    const int per_band = mt * kPBand, band = i / per_band, in = i - band * per_band;
    const int width = min(kPBand, nt - band * kPBand);
    m0 = (in / width) * 256;
    n0 = (band * kPBand + in % width) * 256;
  };
  if (t == 0) {
    for (int i = 0; i < kPStages; ++i) { umma::mbar_init(&full[i], 1); umma::mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { umma::mbar_init(&accFull[i], 1); umma::mbar_init(&accEmpty[i], 8); }   // four epilogue warps in each CTA
    umma::mbar_fence_init();
    dead = (umma::smem_u32(sm) & 1023u) != 0;                           // the swizzled tiles need 1 KB boundaries
    if (dead) g_proj_gemm_status = 1;
    prefetch_map(&xmap);
    prefetch_map(&wmap);
  }
  if (w == 1) {
    umma::pair_tmem_alloc(&tmem_slot, 512);
  }
  umma::fence_before_sync();
  cluster.sync();                                                       // both CTAs' barriers are ready
  umma::fence_after_sync();
  pdl_release();
  pdl_wait();
  const uint32_t tm = tmem_slot;
  bool gave_up = dead;
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if (gave_up) return;
    if (!umma::mbar_wait_timed(bar, parity, &dead)) { gave_up = true; dead = 1; g_proj_gemm_status = 1; }
  };

  if (w == 0) {
    // ---------------------------------------------------------------- producer (each CTA its own rows of X and of W)
    if (l == 0) {
      int it = 0;
      for (int i = pair; i < tiles && !gave_up; i += pairs) {
        int m0, n0;
        tile_at(i, m0, n0);
        for (int kb = 0; kb < kb_n; ++kb, ++it) {
          const int s = it % kPStages;
          if (it >= kPStages) wait(&empty[s], ((it - kPStages) / kPStages) & 1);
          if (gave_up) break;
          unsigned char* st = sm + s * kPStageBytes;
          if (rank == 0) umma::mbar_expect_tx(&full[s], 2 * kPStageBytes);
          const uint32_t bar = umma::cluster_addr(&full[s], 0);
          pair_load_box_2d(st, &xmap, kb * kGK, m0 + 128 * (int)rank, bar);
          pair_load_box_2d(st + kTileBytes, &wmap, kb * kGK, n0 + 128 * (int)rank, bar);
        }
      }
    }
  } else if (w == 1) {
    // ---------------------------------------------------------------- issuer
    if (l == 0 && rank == 0) {
      constexpr uint32_t idesc = idesc_bf16(256, 256);
      int it = 0, local = 0;
      for (int i = pair; i < tiles && !gave_up; i += pairs, ++local) {
        const int acc = local & 1;
        if (local >= 2) wait(&accEmpty[acc], ((local - 2) >> 1) & 1);      // both epilogues have read this accumulator
        umma::fence_after_sync();
        for (int kb = 0; kb < kb_n && !gave_up; ++kb, ++it) {
          const int s = it % kPStages;
          wait(&full[s], (it / kPStages) & 1);
          if (gave_up) break;
          umma::fence_after_sync();
          const unsigned char* st = sm + s * kPStageBytes;
#pragma unroll
          for (int ks = 0; ks < kGK / 16; ++ks)
            umma::pair_mma(tm + acc * 256, tma::desc_sw128(st + ks * 32, 16, 1024), tma::desc_sw128(st + kTileBytes + ks * 32, 16, 1024), idesc,
                     (kb > 0 || ks > 0) ? 1u : 0u);
          umma::pair_commit(&empty[s]);                                           // the stage is free in both CTAs once these MMAs have read it
        }
        if (!gave_up) umma::pair_commit(&accFull[acc]);
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue: warp w owns TMEM lanes 32 (w % 4) .. +31
    const int q = w & 3;
    int local = 0;
    for (int i = pair; i < tiles; i += pairs, ++local) {
      int m0, n0;
      tile_at(i, m0, n0);
      const int acc = local & 1;
      if (l == 0) wait(&accFull[acc], (local >> 1) & 1);
      __syncwarp();
      if (dead) break;
      umma::fence_after_sync();
      const int row = m0 + 128 * (int)rank + 32 * q + l;
#pragma unroll 1
      for (int c = 0; c < 8; ++c) {
        float v[32];
        umma::tmem_ld32(umma::tmem_addr(tm, q, acc * 256 + 32 * c), v);     // warp-collective
        const int col = n0 + 32 * c;
        if (row < P.R && col < P.N) store_chunk(P, row, col, v);
      }
      umma::fence_before_sync();
      __syncwarp();
      if (l == 0) umma::pair_arrive(umma::cluster_addr(&accEmpty[acc], 0));
    }
  }
  umma::fence_before_sync();
  __syncwarp();
  cluster.sync();                                                          // neither CTA leaves while the other may still use its memory
  if (w == 1) umma::pair_tmem_dealloc(tm, 512);
}

// ---- few rows: 128 x TN tiles, K split over a cluster ----------------------------------------------------------------
// A stage holds the rows of X that exist (a multiple of 8, 128 at most) and TN rows of W; as many stages as fit, so that
// a few rows leave the room, and the copy engine, to W.  The MMA reads 128 rows all the same: whatever lies behind the last
// row ends in accumulator rows that nobody stores, and kSRing keeps a whole tile behind the last stage's start.
constexpr int kSRing = 212992, kSMaxStages = 16;
template <int TN> constexpr int kSLd = TN + 4;                           // floats per row of a partial tile in shared memory
constexpr size_t kSplitSmem = (size_t)kSRing + (2 * kSMaxStages + 1) * 8 + 16;
constexpr int kSThreads = 64 + 256;                                       // producer, issuer, eight epilogue warps
template <int TN> constexpr int kTmemCols = TN <= 64 ? 64 : (TN <= 128 ? 128 : 256);

// grid: tiles x splits, cluster = splits (along x); columns fastest inside a band of row tiles.
template <int TN>
__global__ void __launch_bounds__(kSThreads, 1)
proj_gemm_split_kernel(const __grid_constant__ ProjParams P, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, int splits,
                       int xrows, int ST) {
  static_assert(128 * kSLd<TN> * 4 <= kSRing, "the partial tile takes the place of the stages");
  extern __shared__ __align__(1024) unsigned char sm[];
  const int xbytes = xrows * kGK * 2, stage = xbytes + TN * kGK * 2;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + kSRing);
  uint64_t *full = bars, *empty = bars + kSMaxStages, *accFull = bars + 2 * kSMaxStages;
  uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 2 * kSMaxStages + 1);
  volatile int& dead = *reinterpret_cast<volatile int*>(&tmem_slot + 1);
  const int t = threadIdx.x, w = t >> 5, l = t & 31;
  const int mt = (P.R + kGM - 1) / kGM, tile = blockIdx.x / splits, split = blockIdx.x % splits;
  const int m0 = (tile % mt) * kGM, n0 = (tile / mt) * TN;                // row tiles of one W tile side by side
  const int kb_all = P.K / kGK, kb0 = kb_all * split / splits, kb_n = kb_all * (split + 1) / splits - kb0;
  if (t == 0) {
    for (int i = 0; i < ST; ++i) { umma::mbar_init(&full[i], 1); umma::mbar_init(&empty[i], 1); }
    umma::mbar_init(accFull, 1);
    umma::mbar_fence_init();
    dead = (umma::smem_u32(sm) & 1023u) != 0;
    if (dead) g_proj_gemm_status = 1;
    prefetch_map(&xmap);
    prefetch_map(&wmap);
  }
  if (w == 1) umma::tmem_alloc(&tmem_slot, kTmemCols<TN>);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  pdl_release();
  pdl_wait();
  const uint32_t tm = tmem_slot;
  bool gave_up = dead;
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if (gave_up) return;
    if (!umma::mbar_wait_timed(bar, parity, &dead)) { gave_up = true; dead = 1; g_proj_gemm_status = 1; }
  };
  if (w == 0) {
    if (l == 0) {
      for (int it = 0, s = 0, phase = 1; it < kb_n; ++it) {
        if (it >= ST) wait(&empty[s], phase);
        if (gave_up) break;
        unsigned char* st = sm + s * stage;
        umma::mbar_expect_tx(&full[s], stage);
        load_box_2d(st + xbytes, &wmap, (kb0 + it) * kGK, n0, &full[s]);
        load_box_2d(st, &xmap, (kb0 + it) * kGK, m0, &full[s]);
        if (++s == ST) { s = 0; phase ^= 1; }
      }
    }
  } else if (w == 1) {
    if (l == 0) {
      constexpr uint32_t idesc = idesc_bf16(kGM, TN);
      for (int it = 0, s = 0, phase = 0; it < kb_n; ++it) {
        wait(&full[s], phase);
        if (gave_up) break;
        umma::fence_after_sync();
        const unsigned char* st = sm + s * stage;
#pragma unroll
        for (int ks = 0; ks < kGK / 16; ++ks)
          umma::mma_f16_ss(tm, tma::desc_sw128(st + ks * 32, 16, 1024), tma::desc_sw128(st + xbytes + ks * 32, 16, 1024), idesc, (it > 0 || ks > 0) ? 1u : 0u);
        umma::commit(&empty[s]);
        if (++s == ST) { s = 0; phase ^= 1; }
      }
      if (!gave_up) umma::commit(accFull);
    }
  } else {
    const int q = w & 3, r = 32 * q + l;
    if (l == 0) wait(accFull, 0);
    __syncwarp();
    umma::fence_after_sync();
    if (!dead) {
#pragma unroll 1
      for (int c = (w - 2) >> 2; c < TN / 32; c += 2) {                     // the two warps of a lane quarter take every other chunk
        float v[32];
        umma::tmem_ld32(umma::tmem_addr(tm, q, 32 * c), v);                 // warp-collective
        if (splits == 1) {
          if (m0 + r < P.R && n0 + 32 * c < P.N) store_chunk(P, m0 + r, n0 + 32 * c, v);
        } else {                                                            // the stages have been read: the partial tile goes over them
          float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(sm) + (size_t)r * kSLd<TN> + 32 * c);
#pragma unroll
          for (int k = 0; k < 8; ++k) dst[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
        }
      }
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (w == 1) umma::tmem_dealloc(tm, kTmemCols<TN>);
  if (splits == 1) return;
  // Every CTA of the cluster sums a slice of the rows over all partial tiles.
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const int live = min(kGM, P.R - m0), r0 = live * split / splits, r1 = live * (split + 1) / splits;
  constexpr int kQuads = TN / 4, kFlight = 3;
  const float* part[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) part[k] = cluster.map_shared_rank(reinterpret_cast<float*>(sm), k < splits ? k : 0);
  for (int i0 = t; i0 < (r1 - r0) * kQuads; i0 += kFlight * kSThreads) {
    float4 x[kFlight][8];
#pragma unroll
    for (int f = 0; f < kFlight; ++f) {
      const int i = i0 + f * kSThreads;
      const size_t at = (size_t)(r0 + i / kQuads) * kSLd<TN> + (i % kQuads) * 4;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k < splits && i < (r1 - r0) * kQuads) x[f][k] = *reinterpret_cast<const float4*>(part[k] + at);
    }
#pragma unroll
    for (int f = 0; f < kFlight; ++f) {
      const int i = i0 + f * kSThreads, c = (i % kQuads) * 4;
      if (i >= (r1 - r0) * kQuads || n0 + c >= P.N) continue;
      float4 sum = x[f][0];
#pragma unroll
      for (int k = 1; k < 8; ++k)
        if (k < splits) { sum.x += x[f][k].x; sum.y += x[f][k].y; sum.z += x[f][k].z; sum.w += x[f][k].w; }
      store_quad(P, m0 + r0 + i / kQuads, n0 + c, sum);
    }
  }
  cluster.sync();                                                          // the partial tiles stay until everybody has read them
}

// Row-major bf16 matrix [rows][K] as a tensor map with boxes of box_rows x 64 channels, 128-byte swizzle.
static cr_status map_rows_bf16(CUtensorMap* map, const void* base, long long rows, int K, int box_rows) {
  tma::EncodeFn enc;
  if (cr_status s = tma::encoder(&enc)) return s;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kGK, (cuuint32_t)box_rows}, unit[2] = {1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, unit, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed with code %d", (int)r);
    return CR_ERR_CUDA;
  }
  return CR_OK;
}

// How a product is cut.  Costs in cycles: a K step of 16 from its shared-memory traffic (see the head of this file; below
// 128 columns the copy engine's pace), and what a tile's first loads, its epilogue and the sum over a cluster take beside it.
// Every cut was timed on twelve shapes from 1 to 1,500 rows; the choice is within 8 % of the fastest cut on all of them.
// A split has to fit in one wave: clusters of three leave 13 of 148 SMs idle, of eight 28 (a processing cluster holds
// whole thread-block clusters only), and one cluster too many doubles the time, so the room is asked of the runtime.
struct GemmShape { int tn, splits; };                                      // tn 0: CTA pairs
static cr_status cluster_slots(const int (**slots)[9]) {
  static PerDeviceOnce looked_up;
  static int table[64][9];
  int dev = 0;
  CR_CUDA(cudaGetDevice(&dev));
  if (cr_status st = once_per_device(looked_up, [dev] {
        CR_CUDA(cudaFuncSetAttribute(proj_gemm_split_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSplitSmem));
        for (int s = 1; s <= 8; ++s) {
          cudaLaunchConfig_t cfg = {};
          cfg.gridDim = dim3(s); cfg.blockDim = dim3(kSThreads); cfg.dynamicSmemBytes = kSplitSmem;
          cudaLaunchAttribute attr[1];
          attr[0].id = cudaLaunchAttributeClusterDimension;
          attr[0].val.clusterDim.x = s; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
          cfg.attrs = attr; cfg.numAttrs = 1;
          CR_CUDA(cudaOccupancyMaxActiveClusters(&table[dev & 63][s], proj_gemm_split_kernel<128>, &cfg));
        }
        return CR_OK;
      })) return st;
  *slots = &table[dev & 63];
  return CR_OK;
}
static GemmShape gemm_shape(int R, int K, int N, int sms, const int (&slots)[9]) {
  auto up = [](long long a, long long b) { return (a + b - 1) / b; };
  const long long steps = K / 16;
  GemmShape best{0, 1};
  double cost = (double)up(up(R, 256) * up(N, 256), sms / 2) * steps * 133 + 5000;
  const int tns[4] = {64, 96, 128, 256};
  const double step[4] = {96, 112, 132, 195};
  for (int i = 0; i < 4; ++i) {
    const long long tiles = up(R, kGM) * up(N, tns[i]);
    for (int s = 1; s <= 8 && s * 4 <= K / kGK; ++s) {
      if (s > 1 && tiles > slots[s]) break;                                 // splitting pays only while SMs would idle
      const double c = (double)up(tiles * s, sms) * (up(K / kGK, s) * 4 * step[i] + 3000 + tns[i] * 10 + (s > 1 ? 2500 : 0));
      if (c < cost) { cost = c; best = GemmShape{tns[i], s}; }
    }
  }
  return best;
}

template <int TN>
static cr_status split_launch(const ProjParams& P, const CUtensorMap& xmap, const CUtensorMap& wmap, int splits, int xrows, cudaStream_t stream) {
  static PerDeviceOnce configured;
  if (cr_status st = once_per_device(configured, [] {
        CR_CUDA(cudaFuncSetAttribute(proj_gemm_split_kernel<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSplitSmem));
        return CR_OK;
      })) return st;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(((P.R + kGM - 1) / kGM) * ((P.N + TN - 1) / TN) * splits);
  cfg.blockDim = dim3(kSThreads);
  cfg.dynamicSmemBytes = kSplitSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (pdl_enabled()) { attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[na++].val.programmaticStreamSerializationAllowed = 1; }
  if (splits > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = splits; attr[na].val.clusterDim.y = 1; attr[na++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr; cfg.numAttrs = na;
  const int stage = (xrows + TN) * kGK * 2, fit = (kSRing - (stage < kTileBytes ? kTileBytes - stage : 0)) / stage;
  CR_CUDA(cudaLaunchKernelEx(&cfg, proj_gemm_split_kernel<TN>, P, xmap, wmap, splits, xrows, fit < kSMaxStages ? fit : kSMaxStages));
  CR_LAUNCH_CHECK("proj_gemm_split_kernel");
  return CR_OK;
}
}  // namespace cr

extern "C" cr_status cr_proj_gemm(const void* x, const void* w, int R, int K, int N, const cr_proj_out* outs, int n_outs, void* stream_) {
  using namespace cr;
  CR_REQUIRE(x && w && outs, "cr_proj_gemm: null buffer");
  CR_REQUIRE(R >= 1 && N >= 32 && K >= kGK && K % kGK == 0, "cr_proj_gemm: R >= 1, N >= 32, K a multiple of 64 (got R=%d K=%d N=%d)", R, K, N);
  CR_REQUIRE(n_outs >= 1 && n_outs <= kMaxOuts, "cr_proj_gemm: 1..%d outputs", kMaxOuts);
  CR_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)w & 15) == 0, "cr_proj_gemm: operands must be 16-byte aligned");
  ProjParams P;
  P.R = R; P.K = K; P.N = N; P.n_outs = n_outs;
  int next = 0;
  for (int i = 0; i < n_outs; ++i) {
    const cr_proj_out& o = outs[i];
    CR_REQUIRE(o.ptr && o.col0 == next && o.cols >= 32 && o.cols % 32 == 0, "cr_proj_gemm: output %d must start at column %d and hold a multiple of 32 columns", i, next);
    CR_REQUIRE(o.ld >= o.cols && (o.ld * (o.f32 ? 4 : 2)) % 16 == 0 && ((uintptr_t)o.ptr & 15) == 0, "cr_proj_gemm: output %d: row pitch and base must keep 16-byte alignment", i);
    P.ptr[i] = o.ptr; P.col0[i] = o.col0; P.cols[i] = o.cols; P.ld[i] = o.ld; P.f32[i] = o.f32 ? 1 : 0;
    next += o.cols;
  }
  CR_REQUIRE(next == N, "cr_proj_gemm: the outputs cover %d columns, the product has %d", next, N);
  const int(*slots)[9];
  if (cr_status st = cluster_slots(&slots)) return st;
  const GemmShape shape = gemm_shape(R, K, N, sm_count(), *slots);
  CUtensorMap xmap, wmap;
  const int xrows = shape.tn && R < kGM ? (R + 7) / 8 * 8 : kGM;           // rows of a box of X
  if (cr_status st = map_rows_bf16(&xmap, x, R, K, xrows)) return st;
  if (cr_status st = map_rows_bf16(&wmap, w, N, K, shape.tn ? shape.tn : 128)) return st;
  cudaStream_t stream = (cudaStream_t)stream_;
  use_stream(stream);
  if (shape.tn == 64) return split_launch<64>(P, xmap, wmap, shape.splits, xrows, stream);
  if (shape.tn == 96) return split_launch<96>(P, xmap, wmap, shape.splits, xrows, stream);
  if (shape.tn == 128) return split_launch<128>(P, xmap, wmap, shape.splits, xrows, stream);
  if (shape.tn == 256) return split_launch<256>(P, xmap, wmap, shape.splits, xrows, stream);
  static PerDeviceOnce configured;
  if (cr_status st = once_per_device(configured, [] {
        CR_CUDA(cudaFuncSetAttribute(proj_gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairSmem));
        return CR_OK;
      })) return st;
  const int tiles = ((R + 255) / 256) * ((N + 255) / 256), pairs = sm_count() / 2;
  CR_CUDA(launch_pdl(proj_gemm_pair_kernel, dim3(2 * (tiles < pairs ? tiles : pairs)), dim3(kGThreads), kPairSmem, stream, P, xmap, wmap));
  CR_LAUNCH_CHECK("proj_gemm_pair_kernel");
  return CR_OK;
}

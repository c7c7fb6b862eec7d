// QSA prefill attention over row tiles on tcgen05 tensor cores (sm_100a): the job of QsaUnionBuildKernel +
// QsaUnionStageKernel (engine/layers/kernels/prefill_qsa_union.h:25-68, :519-742).
//
// A tile is RT = 128 / gqa consecutive query rows (16 at 8 query heads per KV head, 10 at 12).  The rows of a tile
// share one key list, the union of their attended blocks, so every K/V row is fetched once per tile, and the tile's
// rows x heads are the 128 M rows of the tensor-core products.  A per-block row mask keeps every row's own selection
// exact, and the causal rule (key position <= row position) cuts the tail block.
//
// qsa_union_build_kernel (one CTA per tile): every row contributes its selected blocks (or all complete blocks when
// dense) plus its open tail block to a bitmap over the block ids; ranks in the bitmap are places in the list, where the
// rows OR their bits.  The bitmap is walked in windows, so the context length does not limit it (the reference keeps a
// byte per block in 64 KB of LDS and falls back to row-wise attention past about 196K positions,
// engine/layers/qsa_union_lds.h:7-11).
//
// qsa_flash_tc_kernel (one CTA per (tile, KV head, split), 16 warps, 64 keys per step):
//   loader warps (6)   one per K stage and per V stage: gathers the rows of 16 blocks with 16-byte cp.async, one key's 512
//                      bytes per instruction.  Tiles land as four groups of 64 channels, [64 keys][128 bytes] with the
//                      128-byte swizzle: for K the K-major operand [key][channel], for V the MN-major operand
//                      [key][channel], so neither is transposed anywhere.  The V loaders also build the visibility words.
//   issuer warps (2)   S = Q K^T (16 tcgen05.mma kind::f16, M 128 x N 64 x K 16, the query tile being the A operand
//                      in tensor memory, which leaves the shared memory to the K/V stages) into one of two TMEM
//                      accumulators; O += P V (4 MMAs, N 256) once the probabilities are written.
//   softmax warps (8)  two warpgroups that take the steps in turn, thread = (row, head) = TMEM lane: reads S, applies mask
//                      and causality (two 32-bit visibility words per step), keeps a reference maximum that moves only
//                      when a logit exceeds it by more than 2^8 (the accumulator is rescaled in TMEM then, which is rare
//                      after the first steps), writes P as fp16 into a K-major shared-memory tile, sums it.
//   epilogue           all warps: O through shared memory to a warp per (row, head), / sum, optional un-gated context,
//                      sigmoid gate, output format.
// Bound: the tensor pipe beside the traffic of shared memory (a step takes 2,060 cycles; its 20 MMAs alone 1,550, and the 160 KB
// that the gathers, P and the operands move through shared memory 1,280).  What it took to get there from 3,750: instruction
// fetches were a third of all stalls while the roles had long unrolled bodies (rolled loops), the visibility words sat in the K
// loaders' path (2,600 cycles), a thread wrote a row of its own at the end (20 us per CTA, now 12), and an S accumulator was held
// until the step's exponentials were done, so that the next product into it waited 2,300 cycles for 64 logits that registers
// hold (2,350 cycles a step; what had spilled there was the rescaling of O, 32 columns at a time).  2,048 rows at 30,720, 24
// heads: 406 + 28 us of output transform, 353 us with it, 320 us now.
// q and P are fp16 with fp32 accumulation, the reference's prefill numerics (prefill_qsa_union.h:680-684).
// Every wait is bounded; a wait that gives up raises the status word and the CTA runs to its end.
#include <climits>
#include "qsa.cuh"
#include "tma.cuh"
#include "umma.cuh"

namespace cr {

CR_DEFINE_STATUS_WORD(qsa_flash)

constexpr int kFlKeys = 64;                         // keys per step
constexpr int kFlBlocks = kFlKeys / 4;              // union entries per step
constexpr int kFlStages = 3;                        // K tiles and V tiles in flight, each with a loader warp of its own
constexpr int kFlSeen = 8;                          // steps whose visibility words are kept (a V loader runs at most 6 steps ahead)
constexpr int kFlSoftmax = 8;                       // softmax warps: two warpgroups that take the steps in turn
constexpr int kFlThreads = 32 * (kFlSoftmax + 2 * kFlStages + 2);   // + a loader warp per K and per V stage + an issuer warp per product
constexpr int kFlIssuer = kFlSoftmax + 2 * kFlStages;
constexpr int kFlKBytes = kFlKeys * 256 * 2;        // [4 channel groups][64 keys][128 bytes, 128-byte swizzle]
constexpr int kFlGroup = kFlKeys * 128;             // one channel group of a tile
constexpr int kFlOutLd = 260;                       // floats per (row, head) of the output image in shared memory
constexpr int kFlPBytes = 128 * kFlKeys * 2;        // [8 key pieces][128 rows][8 halves]
constexpr size_t kFlashSmem = 2 * kFlStages * kFlKBytes + 2 * kFlPBytes;   // + 3 KB of static arrays: all of the 227 KB
// TMEM columns: O 0-255, S of step j at 256 + 64 (j & 1), the query tile (two fp16 channels per column) at 384-511
constexpr uint32_t kColO = 0, kColS = 256, kColQ = 384;

struct FlashParams {
  cr_qsa_args a;          // the output rows (pos0 = position of row 0)
  const __half* q_hi;     // [R][Hq][256]
  const int2* list;       // [tiles][cap] (block, row mask), ascending blocks
  const int* count;       // [tiles]
  float* partials;        // splits > 1: records (m, l, acc[256]) [split][R][Hq][258] for the merge kernel, else null
  int cap, RT, Hq, Hkv, fmt;
  int flash_max;          // entries per row of a tile: longer lists are left to the row-wise kernel,
  int flash_mixed;        // as QsaParams::tile_mixed
};

int qsa_union_rows(const cr_geometry* g) {
  const int most = 128 / (g->q_heads / g->kv_heads);
  const int want = options().qsa_union_rows;
  return want > 0 && want < most ? want : most;
}
int qsa_union_cap(int RT) { return (RT * 513 + 15) / 16 * 16; }

// ---- union lists -------------------------------------------------------------------------------------------
// One CTA per tile, a warp per row.  The attended blocks of all rows set bits of a shared-memory bitmap over the block
// ids; a prefix sum of the word popcounts gives every block its rank in the ascending union, and the rows then OR their
// bit into the mask of that rank.  Contexts past kUbWindow blocks (1 M positions) are walked in windows of that many.
// Bound: latency of four short shared-memory passes.  2,048 rows at 262,144 positions: 113 us as a bitonic sort of 8,208
// (block, row) keys (105 barrier-separated passes over 64 KB), 8 us as bitmap + rank.
constexpr int kUbThreads = 512;
constexpr int kUbWindow = 262144;                      // blocks per window: 32 KB of bitmap, 32 KB of word ranks

static size_t union_smem_bytes(int words, int cap) { return ((size_t)2 * words + 2 * (size_t)cap) * sizeof(unsigned); }

__global__ void __launch_bounds__(kUbThreads) qsa_union_build_kernel(const __grid_constant__ cr_qsa_args a, int2* list, int* count, int cap, int RT,
                                                                     int words) {
  extern __shared__ __align__(16) unsigned ub[];
  unsigned* bits = ub;                                   // words: which blocks of the window any row attends
  unsigned* rank = bits + words;                         // words: blocks of the window below this word
  unsigned* mask = rank + words;                         // cap: row bits of the union's entries
  unsigned* ids = mask + cap;                            // cap: their block ids
  __shared__ unsigned red[kUbThreads / 32 + 1];
  const int t = threadIdx.x, w = t >> 5, l = t & 31;
  const int tile = blockIdx.x, row0 = tile * RT, rows = min(RT, a.R - row0);
  const int total = (a.pos0 + row0 + rows - 1) / 4 + 1;  // blocks up to the one of the tile's last row
  // this warp's row (16 warps, at most 16 rows)
  const bool have = w < rows;
  const int gr = row0 + w, p = a.pos0 + gr, nb = (p + 1) / 4;
  const int ns = have ? a.nsel[gr] : 0;
  const int n = have ? (ns < 0 ? nb : CR_SEL_BLOCKS) : 0;   // dense rows attend every complete block (at most 512 of them)
  const int* sel = a.sel + (size_t)gr * CR_SEL_BLOCKS;
  constexpr int kPer = CR_SEL_BLOCKS / 32;
  int blk[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int i = l + 32 * k;
    blk[k] = i < n ? (ns < 0 ? i : sel[i]) : -1;
  }
  const int open = have && (p + 1) % 4 != 0 ? nb : -1;     // the open block holds the tail tokens
  for (int i = t; i < 2 * cap; i += kUbThreads) mask[i] = 0u;
  unsigned base = 0;                                       // entries of the windows before this one
  for (int w0 = 0; w0 < total; w0 += kUbWindow) {
    const int span = min(kUbWindow, total - w0), nw = (span + 31) >> 5;
    auto in_window = [&](int b) { return b >= w0 && b - w0 < span; };
    for (int i = t; i < nw; i += kUbThreads) bits[i] = 0u;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kPer; ++k)
      if (in_window(blk[k])) atomicOr(&bits[(blk[k] - w0) >> 5], 1u << (blk[k] & 31));
    if (l == 0 && in_window(open)) atomicOr(&bits[(open - w0) >> 5], 1u << (open & 31));
    __syncthreads();
    const int per = (nw + kUbThreads - 1) / kUbThreads, i0 = min(t * per, nw), i1 = min(i0 + per, nw);
    unsigned mine = 0;
    for (int i = i0; i < i1; ++i) mine += __popc(bits[i]);
    unsigned inc = mine;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const unsigned o = __shfl_up_sync(0xffffffffu, inc, s);
      if (l >= s) inc += o;
    }
    if (l == 31) red[w] = inc;
    __syncthreads();
    if (w == 0) {
      const unsigned v = l < kUbThreads / 32 ? red[l] : 0u;
      unsigned winc = v;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const unsigned o = __shfl_up_sync(0xffffffffu, winc, s);
        if (l >= s) winc += o;
      }
      if (l < kUbThreads / 32) red[l] = winc - v;
      if (l == 31) red[kUbThreads / 32] = winc;
    }
    __syncthreads();
    unsigned at = base + red[w] + inc - mine;
    for (int i = i0; i < i1; ++i) { rank[i] = at; at += __popc(bits[i]); }
    base += red[kUbThreads / 32];
    __syncthreads();
    auto place = [&](int b) {
      const int word = (b - w0) >> 5;
      const unsigned r = rank[word] + __popc(bits[word] & ((1u << (b & 31)) - 1u));
      atomicOr(&mask[r], 1u << w);
      ids[r] = (unsigned)b;
    };
#pragma unroll
    for (int k = 0; k < kPer; ++k)
      if (in_window(blk[k])) place(blk[k]);
    if (l == 0 && in_window(open)) place(open);
    __syncthreads();
  }
  int2* out = list + (size_t)tile * cap;
  for (int i = t; i < (int)base; i += kUbThreads) out[i] = make_int2((int)ids[i], (int)mask[i]);
  if (t == 0) count[tile] = (int)base;
}

// ---- flash ---------------------------------------------------------------------------------------------------
__device__ __forceinline__ void fl_cp_async16(unsigned d, const void* src, bool valid) {
  const int bytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes));
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ void fl_mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(umma::smem_u32(bar)) : "memory");
}

// grid (Hkv, tiles, splits).  HKV: the cache's KV heads where they are two (row pitches become constants), else 0.
template <int HKV>
__global__ void __launch_bounds__(kFlThreads, 1) qsa_flash_tc_kernel(const __grid_constant__ FlashParams P) {
  extern __shared__ __align__(1024) unsigned char sm[];
  unsigned char* Ks = sm;                                // kFlStages stages
  unsigned char* Vs = Ks + kFlStages * kFlKBytes;        // kFlStages stages
  unsigned char* Ps = Vs + kFlStages * kFlKBytes;        // two buffers
  __shared__ __align__(8) uint64_t bars[4 * kFlStages + kFlSeen + 6];
  __shared__ unsigned seen_s[kFlSeen][16][2];            // per step and row of the tile: which of the step's 64 keys the row sees
  __shared__ float ref_s[2][128];                        // [step parity][lane]: reference maximum after the step
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int dead;
  uint64_t *kFull = bars, *kEmpty = kFull + kFlStages, *vFull = kEmpty + kFlStages, *pvDone = vFull + kFlStages, *seenFull = pvDone + kFlStages;
  uint64_t *sFull = seenFull + kFlSeen, *sEmpty = sFull + 2, *pFull = sEmpty + 2;
  const cr_qsa_args& a = P.a;
  const int t = threadIdx.x, w = t >> 5, l = t & 31;
  // Newest tiles first: their lists are the longest while rows are dense, and the last wave should hold the short ones.
  const int tile = (int)(gridDim.y - 1 - blockIdx.y), g = blockIdx.x, row0 = tile * P.RT;
  const int gqa = P.Hq / P.Hkv;
  const int cnt = P.count[tile];
  const int n_all = (cnt + kFlBlocks - 1) / kFlBlocks;   // steps of the tile; this CTA's share is [step0, step0 + n)
  if (n_all == 0 || !qsa_tile_shares(P.count, tile, P.RT, a.R, P.flash_max, P.flash_mixed)) return;           // a tile without rows, or one the row-wise kernels serve
  const int step0 = (int)((long long)n_all * blockIdx.z / gridDim.z), n = (int)((long long)n_all * (blockIdx.z + 1) / gridDim.z) - step0;
  if ((umma::smem_u32(sm) & 1023u) != 0) {               // the swizzled tiles need their atoms on 1 KB boundaries
    if (t == 0) g_qsa_flash_status = 1;
    return;
  }
  const int last_pos = a.pos0 + a.R - 1;                 // newest position the cache holds

  if (t == 0) {
    for (int i = 0; i < kFlStages; ++i) {
      umma::mbar_init(&kFull[i], 1);                     // the loader warp of the stage
      umma::mbar_init(&vFull[i], 1);
      umma::mbar_init(&kEmpty[i], 1);                    // S of the stage's step has completed
      umma::mbar_init(&pvDone[i], 1);                    // P V of the stage's step has completed
    }
    for (int i = 0; i < kFlSeen; ++i) umma::mbar_init(&seenFull[i], 1);
    for (int i = 0; i < 2; ++i) {
      umma::mbar_init(&sFull[i], 1);
      umma::mbar_init(&sEmpty[i], kFlSoftmax / 2);       // one arrival per warp of the step's warpgroup
      umma::mbar_init(&pFull[i], kFlSoftmax / 2);
    }
    umma::mbar_fence_init();
    dead = 0;
  }
  if (w == kFlIssuer) umma::tmem_alloc(&tmem_slot, 512);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tm = tmem_slot;
  // The gates of the tile's rows are asked into L2 now: the epilogue reads them with nothing else to do.
  for (int i = t; i < min(P.RT, a.R - row0) * gqa * 8 && !P.partials; i += kFlThreads) {
    const int m = i >> 3;
    asm volatile("prefetch.global.L2 [%0];\n" ::"l"(a.q + ((size_t)(row0 + m / gqa) * P.Hq + g * gqa + m % gqa) * 512 + 256 + (i & 7) * 32));
  }
  // Query tile into tensor memory: M row m = (row m / gqa of the tile, head m % gqa of the group) = TMEM lane m, the
  // 256 fp16 channels of the row as 128 columns (the A operand of S = Q K^T is read from tensor memory).  The rows come
  // in coalesced and pass through the first K stage, swizzled so that a thread can read a row of its own.
  {
    constexpr int kRows = 128 * 32 / kFlThreads;           // rows per warp
    uint4 x[kRows];
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int m = w + i * (kFlThreads / 32), r = m / gqa, hq = m % gqa;
      x[i] = make_uint4(0u, 0u, 0u, 0u);
      if (r < P.RT && row0 + r < a.R) x[i] = reinterpret_cast<const uint4*>(P.q_hi + ((size_t)(row0 + r) * P.Hq + g * gqa + hq) * 256)[l];
    }
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int m = w + i * (kFlThreads / 32);
      *reinterpret_cast<uint4*>(Ks + m * 512 + ((l ^ (m & 7)) << 4)) = x[i];
    }
  }
  __syncthreads();
  if (w < 4) {
#pragma unroll 1
    for (int c8 = 0; c8 < 4; ++c8) {
      float v[32];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint4 x = *reinterpret_cast<const uint4*>(Ks + t * 512 + (((c8 * 8 + i) ^ (t & 7)) << 4));
        v[4 * i] = __uint_as_float(x.x); v[4 * i + 1] = __uint_as_float(x.y); v[4 * i + 2] = __uint_as_float(x.z); v[4 * i + 3] = __uint_as_float(x.w);
      }
      umma::tmem_st32(umma::tmem_addr(tm, w, kColQ + 32 * c8), v);
    }
    umma::tmem_st_wait();
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  bool gave_up = false;
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if (gave_up) return;
    if (!umma::mbar_wait_timed(bar, parity, &dead)) { gave_up = true; dead = 1; g_qsa_flash_status = 1; }
  };
  auto warp_wait = [&](uint64_t* bar, uint32_t parity) {   // lane 0 polls for the warp
    if (l == 0) wait(bar, parity);
    __syncwarp();
  };

  if (w == kFlIssuer) {
    // ------------------------------------------------------------------ issuer of S = Q K^T
    if (l == 0) {
      constexpr uint32_t idS = umma::idesc_f16(128, kFlKeys, false, false);
      for (int j = 0; j < n; ++j) {
        const int st = j % kFlStages;
        wait(&kFull[st], (j / kFlStages) & 1);
        if (j >= 2) wait(&sEmpty[j & 1], ((j >> 1) - 1) & 1);          // the softmax has read the accumulator's step before
        if (gave_up || dead) break;                                    // no more tensor-core work once any wait has run out
        umma::fence_after_sync();
        const uint64_t dK = tma::desc_sw128(Ks + st * kFlKBytes, 16, 1024);
#pragma unroll
        for (int ks = 0; ks < 16; ++ks)                  // 16 channels per MMA: 8 columns of Q, 32 bytes of every key's 128-byte row
          umma::mma_f16_ts(tm + kColS + 64 * (j & 1), tm + kColQ + 8 * ks, dK + (uint64_t)(((ks >> 2) * kFlGroup + (ks & 3) * 32) >> 4), idS, ks > 0);
        umma::commit(&sFull[j & 1]);
        umma::commit(&kEmpty[st]);
      }
    }
  } else if (w == kFlIssuer + 1) {
    // ------------------------------------------------------------------ issuer of O += P V
    if (l == 0) {
      constexpr uint32_t idO = umma::idesc_f16(128, 256, false, true);
      for (int j = 0; j < n; ++j) {
        const int st = j % kFlStages;
        wait(&vFull[st], (j / kFlStages) & 1);
        wait(&pFull[j & 1], (j >> 1) & 1);
        if (gave_up || dead) break;
        umma::fence_after_sync();
        const uint64_t dP = umma::smem_desc(Ps + (j & 1) * kFlPBytes, 128 * 16, 128);
        const uint64_t dV = tma::desc_sw128(Vs + st * kFlKBytes, kFlGroup, 1024);        // MN-major: 64-channel groups, atoms of 8 keys
#pragma unroll
        for (int kk = 0; kk < kFlKeys / 16; ++kk)
          umma::mma_f16_ss(tm + kColO, dP + (uint64_t)(kk * 2 * 128), dV + (uint64_t)(kk * 2048 >> 4), idO, (j > 0 || kk > 0) ? 1u : 0u);
        umma::commit(&pvDone[st]);
      }
    }
  } else if (w >= kFlSoftmax) {
    // ------------------------------------------------------------------ loaders: a warp per K stage and per V stage
    // One cp.async instruction brings one key's 512 bytes: four full lines, and eight lanes write the eight pieces of a
    // 128-byte swizzled row, so the writes are free of bank conflicts.
    const bool keys = w < kFlSoftmax + kFlStages;
    const int st = (w - kFlSoftmax) % kFlStages;
    const char* base = reinterpret_cast<const char*>(keys ? a.c.k : a.c.v) + (size_t)g * 512 + l * 16;
    uint64_t *full = (keys ? kFull : vFull) + st, *empty = (keys ? kEmpty : pvDone) + st;
    const int2* lst = P.list + (size_t)tile * P.cap;
    const size_t row_bytes = HKV ? (size_t)HKV * 512 : (size_t)P.Hkv * 512;
    const unsigned slot = umma::smem_u32((keys ? Ks : Vs) + st * kFlKBytes) + (l >> 3) * kFlGroup + ((l & 7) << 4);
    auto entry = [&](int j) {                              // lane b (and b + 16): entry b of step j
      const int idx = (step0 + j) * kFlBlocks + (l & 15);
      return j < n && idx < cnt ? lst[idx] : make_int2(0, 0);
    };
    int2 e = entry(st);
    for (int j = st; j < n; j += kFlStages) {
      const int2 e_next = entry(j + kFlStages);            // in flight while the stage is waited for
      if (!keys) {
        // Lane r + 16 h builds half h of the word pair of row r: bit 4 b + k is set when the row's bit of block b's mask is
        // set and token k of the block is not in the row's future (only the open tail block of a row can hold such tokens).
        // The V loaders do this, who would wait for the product before anyway: in a K loader it delayed every step.
        const int row = l & 15, prow = a.pos0 + row0 + row;
        const bool rowok = row < P.RT && row0 + row < a.R;
        unsigned word = 0u;
#pragma unroll 2
        for (int b = 0; b < kFlBlocks / 2; ++b) {
          const int src = (l >> 4) * (kFlBlocks / 2) + b;
          const int blk = __shfl_sync(0xffffffffu, e.x, src), msk = __shfl_sync(0xffffffffu, e.y, src);
          const int lim = prow - blk * 4;                             // tokens 0 .. lim of the block are visible
          const unsigned nib = (rowok && ((msk >> row) & 1)) ? (lim >= 3 ? 0xFu : (lim < 0 ? 0u : (2u << lim) - 1u)) : 0u;
          word |= nib << (4 * b);
        }
        seen_s[j % kFlSeen][row][l >> 4] = word;
        __syncwarp();
        if (l == 0) fl_mbar_arrive(&seenFull[j % kFlSeen]);
      }
      if (j >= kFlStages) warp_wait(empty, ((j - kFlStages) / kFlStages) & 1);
      if (dead) break;
#pragma unroll 1
      for (int b = 0; b < kFlBlocks; b += 2) {               // eight keys: one swizzle atom (small loop bodies: see the softmax)
        const unsigned at = slot + b * 512;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int blk = __shfl_sync(0xffffffffu, e.x, b + h), newest = last_pos - blk * 4;   // tokens 0 .. newest of the block are cached
          const char* src = base + (size_t)blk * (4 * row_bytes);
#pragma unroll
          for (int k = 0; k < 4; ++k) fl_cp_async16((at ^ ((h * 4 + k) << 4)) + (h * 4 + k) * 128, k <= newest ? src + k * row_bytes : base, k <= newest);
        }
      }
      asm volatile("cp.async.commit_group;\n" ::);
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      umma::fence_async_smem();
      __syncwarp();
      if (l == 0) fl_mbar_arrive(full);
      e = e_next;
    }
  } else {
    // ------------------------------------------------------------------ softmax warps: thread = TMEM lane m = (row, head)
    // Warpgroup hf takes the steps hf, hf + 2, ...: while one exponentiates a step the other reads the next.  What passes
    // from step to step is the reference maximum of the lane, through shared memory and a 64-thread named barrier per
    // lane quarter and direction.
    const int m = t & 127, hf = t >> 7, r = m / gqa;
    const int give = 1 + 4 * hf + (w & 3), take = 1 + 4 * (hf ^ 1) + (w & 3);
    constexpr float kScale = 0.0625f * 1.4426950408889634f;            // logits / 16, in powers of two
    float m_ref = -INFINITY, lsum = 0.f;                               // lsum: this warpgroup's steps, relative to m_ref
    for (int j = hf; j < n; j += 2) {
      const int s = j & 1;
      warp_wait(&seenFull[j % kFlSeen], (j / kFlSeen) & 1);
      const unsigned see0 = r < 16 ? seen_s[j % kFlSeen][r][0] : 0u, see1 = r < 16 ? seen_s[j % kFlSeen][r][1] : 0u;
      warp_wait(&sFull[s], (j >> 1) & 1);
      umma::fence_after_sync();
      // The step's 64 logits are read at once and the accumulator is free again: the product of step j + 2 runs beside the rest.
      float sv[kFlKeys];
      umma::tmem_ld64(umma::tmem_addr(tm, w, kColS + 64 * s), sv);
      umma::fence_before_sync();
      __syncwarp();
      if (l == 0) umma::mbar_arrive_relaxed(&sEmpty[s]);
      float tmax = -INFINITY, t1 = -INFINITY;
#pragma unroll
      for (int c = 0; c < 32; ++c) {                                    // keys that the row does not see drop out
        sv[c] = (see0 >> c) & 1u ? sv[c] : -INFINITY;
        sv[32 + c] = (see1 >> c) & 1u ? sv[32 + c] : -INFINITY;
      }
#pragma unroll
      for (int c = 0; c < kFlKeys; c += 4) {
        tmax = max3(tmax, sv[c], sv[c + 1]);
        t1 = max3(t1, sv[c + 2], sv[c + 3]);
      }
      tmax = fmaxf(tmax, t1);
      tmax *= kScale;
      float ref = -INFINITY;                                            // the lane's reference after step j - 1
      if (j > 0) {
        asm volatile("bar.sync %0, 64;\n" ::"r"(take) : "memory");
        ref = ref_s[s ^ 1][m];
      }
      const bool move = tmax > ref + 8.f;                               // also the first visible key (ref = -inf)
      const float nref = move ? tmax : ref;
      ref_s[s][m] = nref;
      if (j + 1 < n) asm volatile("bar.arrive %0, 64;\n" ::"r"(give) : "memory");
      if (m_ref != nref) lsum *= exp2f(m_ref - nref);                    // 0 when nothing was accumulated yet
      m_ref = nref;
      if (j > 0 && __any_sync(0xffffffffu, move)) {                      // O holds the steps before this one
        const float factor = move ? exp2f(ref - nref) : 1.f;
        warp_wait(&pvDone[(j - 1) % kFlStages], ((j - 1) / kFlStages) & 1);
        umma::fence_after_sync();
#pragma unroll 1
        for (int c16 = 0; c16 < 16; ++c16) {                             // 16 columns at a time beside the 64 logits
          float o[16];
          umma::tmem_ld16(umma::tmem_addr(tm, w, kColO + 16 * c16), o);
#pragma unroll
          for (int c = 0; c < 16; ++c) o[c] *= factor;
          umma::tmem_st16(umma::tmem_addr(tm, w, kColO + 16 * c16), o);
        }
        umma::tmem_st_wait();
      }
      if (j >= 2) warp_wait(&pvDone[(j - 2) % kFlStages], ((j - 2) / kFlStages) & 1);   // the MMAs of step j - 2 have read this P buffer
      unsigned char* pd = Ps + s * kFlPBytes;
      const float sub = m_ref == -INFINITY ? 0.f : m_ref;               // nothing visible yet: every key drops out
      f2 add = 0ull;
#pragma unroll
      for (int kc8 = 0; kc8 < kFlKeys / 8; ++kc8) {
        unsigned pk[4];
#pragma unroll
        for (int q2 = 0; q2 < 4; ++q2) {
          const int c = kc8 * 8 + 2 * q2;
          const float p0 = ex2_ftz(fmaf(sv[c], kScale, -sub)), p1 = ex2_ftz(fmaf(sv[c + 1], kScale, -sub));
          add = add2(add, pack2(p0, p1));
          const __half2 hp = __floats2half2_rn(p0, p1);
          pk[q2] = *reinterpret_cast<const unsigned*>(&hp);
        }
        *reinterpret_cast<uint4*>(pd + ((size_t)kc8 * 128 + m) * 16) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
      }
      const float2 both = unpack2(add);
      lsum += both.x + both.y;
      umma::fence_async_smem();
      umma::fence_before_sync();
      __syncwarp();
      if (l == 0) fl_mbar_arrive(&pFull[s]);
    }
    // ---------------------------------------------------------------- epilogue: each warpgroup writes half of the channels
    auto both_sync = [] { asm volatile("bar.sync 9, 256;\n" ::: "memory"); };
    both_sync();
    float* sum_s = reinterpret_cast<float*>(&seen_s[0][0][0]);           // 128 floats: no step reads its words any more
    const float last_ref = n > 0 ? ref_s[(n - 1) & 1][m] : -INFINITY;
    if (m_ref != last_ref) lsum *= exp2f(m_ref - last_ref);
    m_ref = last_ref;
    if (hf == 1) sum_s[m] = lsum;
    both_sync();
    if (hf == 0) { sum_s[m] += lsum; ref_s[(n & 1)][m] = m_ref; }
    if (n > 0) warp_wait(&pvDone[(n - 1) % kFlStages], ((n - 1) / kFlStages) & 1);
    umma::fence_after_sync();
    // O to shared memory (every tile and probability has been read), padded so that neither side has bank conflicts
#pragma unroll 1
    for (int c8 = 4 * hf; c8 < 4 * hf + 4; ++c8) {
      float o[32];
      umma::tmem_ld32(umma::tmem_addr(tm, w, kColO + 32 * c8), o);
      float* dst = reinterpret_cast<float*>(sm) + m * kFlOutLd + 32 * c8;
#pragma unroll
      for (int c = 0; c < 32; c += 4) *reinterpret_cast<float4*>(dst + c) = make_float4(o[c], o[c + 1], o[c + 2], o[c + 3]);
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (w == kFlIssuer) umma::tmem_dealloc(tm, 512);
  if (dead) return;
  // Output rows, a warp per (row, head): lane l holds the channels 4 l .. + 3 and 128 + 4 l .. + 3.
  const float* sums = reinterpret_cast<const float*>(&seen_s[0][0][0]);
  constexpr int kWarps = kFlThreads / 32, kBatch = 4;      // gates of four rows are in flight before the first is used
  const int live = min(P.RT, a.R - row0) * gqa;
#pragma unroll 1
  for (int m0 = w; m0 < live; m0 += kBatch * kWarps) {
    float4 gate[kBatch][2];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int m = m0 + k * kWarps;
      if (m >= live || P.partials) break;
      const float4* src = reinterpret_cast<const float4*>(a.q + ((size_t)(row0 + m / gqa) * P.Hq + g * gqa + m % gqa) * 512 + 256) + l;
      gate[k][0] = src[0]; gate[k][1] = src[32];
    }
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int m = m0 + k * kWarps, gr = row0 + m / gqa, h = g * gqa + m % gqa;
      if (m >= live) break;
      const float4* src = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(sm) + m * kFlOutLd) + l;
      float4 o[2] = {src[0], src[32]};
      const float lsum = sums[m];
      if (P.partials) {                                    // the tile is split: (m, l, acc) of this share
        float* rec = P.partials + (((size_t)blockIdx.z * a.R + gr) * P.Hq + h) * CR_QSA_PART;
        if (l == 0) *reinterpret_cast<float2*>(rec) = make_float2(ref_s[n & 1][m] * 0.6931471805599453f, lsum);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (n == 0) o[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          *reinterpret_cast<float2*>(rec + 2 + 128 * i + 4 * l) = make_float2(o[i].x, o[i].y);
          *reinterpret_cast<float2*>(rec + 4 + 128 * i + 4 * l) = make_float2(o[i].z, o[i].w);
        }
        continue;
      }
      const float inv = 1.f / lsum;
#pragma unroll
      for (int i = 0; i < 2; ++i)
        emit_group(a, P.Hq, gr, h, 128 * i + 4 * l, make_float4(o[i].x * inv, o[i].y * inv, o[i].z * inv, o[i].w * inv), gate[k][i], P.fmt);
    }
  }
}

cr_status qsa_union_build_launch(const cr_geometry* g, const cr_qsa_args& a, int2* list, int* count, cudaStream_t stream) {
  static PerDeviceOnce configured;
  if (cr_status st = once_per_device(configured, [] {
        CR_CUDA(cudaFuncSetAttribute(qsa_union_build_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)union_smem_bytes(kUbWindow / 32, qsa_union_cap(16))));
        return CR_OK;
      })) return st;
  const int RT = qsa_union_rows(g), tiles = (a.R + RT - 1) / RT, cap = qsa_union_cap(RT);
  const int blocks = (a.pos0 + a.R - 1) / 4 + 1, words = ((blocks < kUbWindow ? blocks : kUbWindow) + 31) / 32;
  use_stream(stream);
  qsa_union_build_kernel<<<tiles, kUbThreads, union_smem_bytes(words, cap), stream>>>(a, list, count, cap, RT, words);
  CR_LAUNCH_CHECK("qsa_union_build_kernel");
  return CR_OK;
}

// Attention of the rows of `a` over the union lists; splits > 1 leaves records in `partials` for qsa_merge_launch.
cr_status qsa_flash_launch(const cr_geometry* g, const cr_qsa_args& a, const __half* q_hi, const int2* list, const int* count,
                           float* partials, int splits, cr_out_format fmt, int flash_max, int flash_mixed, cudaStream_t stream) {
  static PerDeviceOnce configured;
  if (cr_status st = once_per_device(configured, [] {
        CR_CUDA(cudaFuncSetAttribute(qsa_flash_tc_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFlashSmem));
        CR_CUDA(cudaFuncSetAttribute(qsa_flash_tc_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFlashSmem));
        return CR_OK;
      })) return st;
  FlashParams P;
  P.a = a; P.q_hi = q_hi; P.list = list; P.count = count;
  P.RT = qsa_union_rows(g); P.cap = qsa_union_cap(P.RT);
  P.Hq = g->q_heads; P.Hkv = g->kv_heads; P.fmt = (int)fmt;
  P.partials = splits > 1 ? partials : nullptr;
  P.flash_max = flash_max; P.flash_mixed = flash_mixed;
  const int tiles = (a.R + P.RT - 1) / P.RT;
  use_stream(stream);
  const dim3 grid(g->kv_heads, tiles, splits);
  if (g->kv_heads == 2) qsa_flash_tc_kernel<2><<<grid, kFlThreads, kFlashSmem, stream>>>(P);
  else qsa_flash_tc_kernel<0><<<grid, kFlThreads, kFlashSmem, stream>>>(P);
  CR_LAUNCH_CHECK("qsa_flash_tc_kernel");
  return CR_OK;
}

}  // namespace cr

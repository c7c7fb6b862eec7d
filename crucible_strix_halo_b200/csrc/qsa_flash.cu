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
// qsa_flash_tc_kernel (one CTA per (tile, KV head), 15 warps, 64 keys per step):
//   loader warps (6)   gather the K and V rows of 16 blocks per step with 16-byte cp.async into three stages, two
//                      warps per stage, one key's 512 bytes per instruction.  Both tiles land as four groups of 64
//                      channels, [64 keys][128 bytes] with the 128-byte swizzle: for K the K-major operand
//                      [key][channel], for V the MN-major operand [key][channel], so neither is transposed anywhere.
//   issuer warp        S = Q K^T (16 tcgen05.mma kind::f16, M 128 x N 64 x K 16, the query tile being the A operand
//                      in tensor memory, which leaves the shared memory to the K/V stages) into one of two TMEM
//                      accumulators, one step ahead of the softmax; O += P V (4 MMAs, N 256) once the probabilities
//                      are written.  An event loop issues whichever is ready.
//   softmax warps (8)  two warps per TMEM lane quarter, thread = (row, head) x half of the step's 64 keys: reads S,
//                      applies mask and causality (a 32-bit visibility word per step), keeps a running reference
//                      maximum that moves only when a logit exceeds it by more than 2^8 (the accumulator is rescaled
//                      in TMEM then, which is rare after the first steps; the two halves agree on the row maximum
//                      through shared memory and a 64-thread named barrier), writes P as fp16 into a K-major
//                      shared-memory tile, sums it.
//   epilogue           O / sum, optional un-gated context, sigmoid gate, output format.
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
constexpr int kFlStages = 3;                        // K/V stages in flight
constexpr int kFlSoftmax = 8;                       // softmax warps: two per TMEM lane quarter, 32 keys of a step each
constexpr int kFlThreads = 32 * (kFlSoftmax + 2 * kFlStages + 1);   // + 2 loader warps per stage + 1 issuer warp
constexpr int kFlIssuer = kFlSoftmax + 2 * kFlStages;
constexpr int kFlKBytes = kFlKeys * 256 * 2;        // [4 channel groups][64 keys][128 bytes, 128-byte swizzle]
constexpr int kFlGroup = kFlKeys * 128;             // one channel group of a tile
constexpr int kFlPBytes = 128 * kFlKeys * 2;        // [8 key pieces][128 rows][8 halves]
constexpr size_t kFlashSmem = 2 * kFlStages * kFlKBytes + 2 * kFlPBytes;   // + 3 KB of static arrays: all of the 227 KB
// TMEM columns: O 0-255, S of step j at 256 + 64 (j & 1), the query tile (two fp16 channels per column) at 384-511
constexpr uint32_t kColO = 0, kColS = 256, kColQ = 384;

struct FlashParams {
  cr_qsa_args a;          // the output rows (pos0 = position of row 0)
  const __half* q_hi;     // [R][Hq][256]
  const int2* list;       // [tiles][cap] (block, row mask), ascending blocks
  const int* count;       // [tiles]
  float* gated;           // gated fp32 [R][Hq * 256] when the output transform runs as a second kernel, else null
  float* partials;        // splits > 1: records (m, l, acc[256]) [split][R][Hq][258] for the merge kernel, else null
  int cap, RT, Hq, Hkv, fmt;
  int flash_max;          // tiles whose union list is longer are left to the row-wise kernels
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
__device__ __forceinline__ void fl_mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(umma::smem_u32(bar)) : "memory");
}

// grid (tiles, Hkv, splits).
__global__ void __launch_bounds__(kFlThreads, 1) qsa_flash_tc_kernel(const __grid_constant__ FlashParams P) {
  extern __shared__ __align__(1024) unsigned char sm[];
  unsigned char* Ks = sm;                                // kFlStages stages
  unsigned char* Vs = Ks + kFlStages * kFlKBytes;        // kFlStages stages
  unsigned char* Ps = Vs + kFlStages * kFlKBytes;        // two buffers
  __shared__ __align__(8) uint64_t bars[2 * kFlStages + 4];
  __shared__ unsigned seen_s[kFlStages][16][2];          // per stage and row of the tile: which of the step's 64 keys the row sees
  __shared__ float half_max[2][2][128];                  // [step parity][half][lane]: exchange between the two warps of a TMEM lane quarter
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int dead;
  uint64_t *kvFull = &bars[0], *pvDone = &bars[kFlStages], *sFull = &bars[2 * kFlStages], *pFull = &bars[2 * kFlStages + 2];
  const cr_qsa_args& a = P.a;
  const int t = threadIdx.x, w = t >> 5, l = t & 31;
  const int tile = blockIdx.x, g = blockIdx.y, row0 = tile * P.RT;
  const int gqa = P.Hq / P.Hkv;
  const int cnt = P.count[tile];
  const int n_all = (cnt + kFlBlocks - 1) / kFlBlocks;   // steps of the tile; this CTA's share is [step0, step0 + n)
  if (n_all == 0 || cnt > P.flash_max) return;           // a tile without rows, or one the row-wise kernels serve
  const int step0 = (int)((long long)n_all * blockIdx.z / gridDim.z), n = (int)((long long)n_all * (blockIdx.z + 1) / gridDim.z) - step0;
  if ((umma::smem_u32(sm) & 1023u) != 0) {               // the swizzled tiles need their atoms on 1 KB boundaries
    if (t == 0) g_qsa_flash_status = 1;
    return;
  }
  const int last_pos = a.pos0 + a.R - 1;                 // newest position the cache holds

  if (t == 0) {
    for (int i = 0; i < kFlStages; ++i) {
      umma::mbar_init(&kvFull[i], 2);                    // the two loader warps of the stage
      umma::mbar_init(&pvDone[i], 1);                    // every MMA that read the stage has completed
    }
    for (int i = 0; i < 2; ++i) {
      umma::mbar_init(&sFull[i], 1);
      umma::mbar_init(&pFull[i], kFlSoftmax);            // one arrival per softmax warp
    }
    umma::mbar_fence_init();
    dead = 0;
  }
  if (w == kFlIssuer) umma::tmem_alloc(&tmem_slot, 512);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tm = tmem_slot;
  // Query tile into tensor memory: M row m = (row m / gqa of the tile, head m % gqa of the group) = TMEM lane m, the
  // 256 fp16 channels of the row as 128 columns (the A operand of S = Q K^T is read from tensor memory).
  if (w < 4) {
    const int m = t, r = m / gqa, hq = m % gqa;
    const bool have = r < P.RT && row0 + r < a.R;
    const uint4* src = reinterpret_cast<const uint4*>(P.q_hi + ((size_t)(have ? row0 + r : 0) * P.Hq + g * gqa + hq) * 256);
#pragma unroll 1
    for (int c8 = 0; c8 < 4; ++c8) {
      float v[32];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint4 x = have ? src[c8 * 8 + i] : make_uint4(0u, 0u, 0u, 0u);
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
    // ------------------------------------------------------------------ issuer
    if (l == 0) {
      constexpr uint32_t idS = umma::idesc_f16(128, kFlKeys, false, false), idO = umma::idesc_f16(128, 256, false, true);
      auto issue_S = [&](int j) {
        const uint64_t dK = tma::desc_sw128(Ks + (j % kFlStages) * kFlKBytes, 16, 1024);
#pragma unroll
        for (int ks = 0; ks < 16; ++ks)                  // 16 channels per MMA: 8 columns of Q, 32 bytes of every key's 128-byte row
          umma::mma_f16_ts(tm + kColS + 64 * (j & 1), tm + kColQ + 8 * ks, dK + (uint64_t)(((ks >> 2) * kFlGroup + (ks & 3) * 32) >> 4), idS, ks > 0);
        umma::commit(&sFull[j & 1]);
      };
      // Event loop: S of step ns (one step ahead of the softmax at most, its accumulator being free once the
      // probabilities of step ns - 2 are written) as soon as its tiles have landed, O += P V of step np as soon as its
      // probabilities are written; neither waits for the other's barrier.
      auto ready = [&](uint64_t* bar, uint32_t parity) { return umma::mbar_try(umma::smem_u32(bar), parity); };
      auto now_ns = [] { uint64_t v; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(v)); return v; };
      int ns = 0, np = 0, idle = 0;
      uint64_t t_idle = 0;
      while (np < n) {
        if (ns < n && ns <= np + 1 && ready(&kvFull[ns % kFlStages], (ns / kFlStages) & 1)) {
          umma::fence_after_sync();
          issue_S(ns);
          ++ns; idle = 0;
        } else if (np < ns && ready(&pFull[np & 1], (np >> 1) & 1)) {
          const int st = np % kFlStages;
          umma::fence_after_sync();
          const uint64_t dP = umma::smem_desc(Ps + (np & 1) * kFlPBytes, 128 * 16, 128);
          const uint64_t dV = tma::desc_sw128(Vs + st * kFlKBytes, kFlGroup, 1024);        // MN-major: 64-channel groups, atoms of 8 keys
#pragma unroll
          for (int kk = 0; kk < kFlKeys / 16; ++kk)
            umma::mma_f16_ss(tm + kColO, dP + (uint64_t)(kk * 2 * 128), dV + (uint64_t)(kk * 2048 >> 4), idO, (np > 0 || kk > 0) ? 1u : 0u);
          umma::commit(&pvDone[st]);
          ++np; idle = 0;
        } else if ((++idle & 63) == 0) {                  // nothing ready: look at the clock now and then
          const uint64_t t1 = now_ns();
          if (idle == 64) t_idle = t1;
          if (dead || t1 - t_idle > 2000000000ull) { dead = 1; g_qsa_flash_status = 1; break; }
        }
      }
    }
  } else if (w >= kFlSoftmax) {
    // ------------------------------------------------------------------ loaders: two warps per stage, half of its keys each
    // One cp.async instruction brings one key's 512 bytes: four full lines, and eight lanes write the eight pieces of a
    // 128-byte swizzled row, so the writes are free of bank conflicts.
    const int st = (w - kFlSoftmax) >> 1, lw = (w - kFlSoftmax) & 1;
    const char* kc = reinterpret_cast<const char*>(a.c.k) + (size_t)g * 512 + l * 16;
    const char* vc = reinterpret_cast<const char*>(a.c.v) + (size_t)g * 512 + l * 16;
    const int2* lst = P.list + (size_t)tile * P.cap;
    const size_t row_bytes = (size_t)P.Hkv * 512;
    const unsigned kd = umma::smem_u32(Ks + st * kFlKBytes) + (l >> 3) * kFlGroup, vd = umma::smem_u32(Vs + st * kFlKBytes) + (l >> 3) * kFlGroup;
    auto entry = [&](int j) {                              // lane b (and b + 16): entry b of step j
      const int idx = (step0 + j) * kFlBlocks + (l & 15);
      return j < n && idx < cnt ? lst[idx] : make_int2(0, 0);
    };
    int2 e = entry(st);
    for (int j = st; j < n; j += kFlStages) {
      const int2 e_next = entry(j + kFlStages);            // in flight while the stage is waited for
      if (j >= kFlStages) warp_wait(&pvDone[st], ((j - kFlStages) / kFlStages) & 1);   // the MMAs of the stage's last step are done
      if (dead) break;
#pragma unroll
      for (int b = 0; b < kFlBlocks / 2; ++b) {
        const int pos0 = __shfl_sync(0xffffffffu, e.x, lw * (kFlBlocks / 2) + b) * 4;
        const size_t src = (size_t)pos0 * row_bytes;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int key = (lw * (kFlBlocks / 2) + b) * 4 + k;
          const bool valid = pos0 + k <= last_pos;
          const size_t at = valid ? src + k * row_bytes : 0;
          const unsigned dst = key * 128 + (((l ^ key) & 7) << 4);
          fl_cp_async16(kd + dst, kc + at, valid);
          fl_cp_async16(vd + dst, vc + at, valid);
        }
      }
      asm volatile("cp.async.commit_group;\n" ::);
      if (lw == 0) {
        // Lane r < 16 builds the word of row r: bit 4 b + k is set when the row's bit of block b's mask is set and token k
        // of the block is not in the row's future (only the open tail block of a row can hold such tokens).  The softmax
        // threads read one word per step.
        const int prow = a.pos0 + row0 + (l & 15);
        const bool rowok = (l & 15) < P.RT && row0 + (l & 15) < a.R;
        unsigned lo_w = 0u, hi_w = 0u;
#pragma unroll
        for (int b = 0; b < kFlBlocks; ++b) {
          const int blk = __shfl_sync(0xffffffffu, e.x, b), msk = __shfl_sync(0xffffffffu, e.y, b);
          const int lim = prow - blk * 4;                             // tokens 0 .. lim of the block are visible
          const unsigned nib = (rowok && ((msk >> (l & 15)) & 1)) ? (lim >= 3 ? 0xFu : (lim < 0 ? 0u : (2u << lim) - 1u)) : 0u;
          if (b < 8) lo_w |= nib << (4 * b); else hi_w |= nib << (4 * (b - 8));
        }
        if (l < 16) { seen_s[st][l][0] = lo_w; seen_s[st][l][1] = hi_w; }
      }
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      umma::fence_async_smem();
      __syncwarp();
      if (l == 0) fl_mbar_arrive(&kvFull[st]);
      e = e_next;
    }
  } else {
    // ------------------------------------------------------------------ softmax warps: thread = (TMEM lane m, half of the step's keys)
    // Warps w and w + 4 share the lanes 32 (w % 4) .. +31; warp w takes the keys 0-31 of a step, warp w + 4 the keys 32-63.
    const int m = t & 127, hf = t >> 7, r = m / gqa, hq = m % gqa;
    const bool rowok = r < P.RT && row0 + r < a.R;
    const int pair_bar = 1 + (w & 3);                                   // named barrier of the two warps of a lane quarter
    auto pair_sync = [&] { asm volatile("bar.sync %0, 64;\n" ::"r"(pair_bar) : "memory"); };
    constexpr float kScale = 0.0625f * 1.4426950408889634f;            // logits / 16, in powers of two
    float m_ref = -INFINITY, lsum = 0.f;
    for (int j = 0; j < n; ++j) {
      const int s = j & 1, st = j % kFlStages;
      warp_wait(&kvFull[st], (j / kFlStages) & 1);                     // block ids and masks of the step are visible
      const unsigned seen = r < 16 ? seen_s[st][r][hf] : 0u;             // which of this thread's 32 keys its row sees
      warp_wait(&sFull[s], (j >> 1) & 1);
      umma::fence_after_sync();
      float sv[32];
      umma::tmem_ld32(umma::tmem_addr(tm, w, kColS + 64 * s + 32 * hf), sv);
      float tmax = -INFINITY;
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        sv[c] = (seen >> c) & 1u ? sv[c] * kScale : -INFINITY;
        tmax = fmaxf(tmax, sv[c]);
      }
      half_max[s][hf][m] = tmax;                                        // (parity: the partner may still be reading the step before)
      pair_sync();
      tmax = fmaxf(tmax, half_max[s][hf ^ 1][m]);                       // the row's maximum over all 64 keys of the step
      const bool move = tmax > m_ref + 8.f;                             // also the first visible key (m_ref = -inf)
      if (__any_sync(0xffffffffu, move)) {
        const float nref = move ? tmax : m_ref;
        const float factor = move ? exp2f(m_ref - nref) : 1.f;          // 0 when nothing was accumulated yet
        lsum *= factor;
        m_ref = nref;
        if (j > 0) {                                                    // O holds the steps before this one; each warp rescales half of it
          warp_wait(&pvDone[(j - 1) % kFlStages], ((j - 1) / kFlStages) & 1);
          umma::fence_after_sync();
#pragma unroll 1
          for (int c8 = 4 * hf; c8 < 4 * hf + 4; ++c8) {
            float o[32];
            umma::tmem_ld32(umma::tmem_addr(tm, w, kColO + 32 * c8), o);
#pragma unroll
            for (int c = 0; c < 32; ++c) o[c] *= factor;
            umma::tmem_st32(umma::tmem_addr(tm, w, kColO + 32 * c8), o);
          }
          umma::tmem_st_wait();
        }
      }
      if (j >= 2) warp_wait(&pvDone[(j - 2) % kFlStages], ((j - 2) / kFlStages) & 1);   // the MMAs of step j - 2 have read this P buffer
      unsigned char* pd = Ps + s * kFlPBytes;
      float add = 0.f;
#pragma unroll
      for (int kc8 = 0; kc8 < 4; ++kc8) {
        unsigned pk[4];
#pragma unroll
        for (int q2 = 0; q2 < 4; ++q2) {
          float p0, p1;                                                // 2^(-inf) = 0: keys the row does not see drop out
          asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p0) : "f"(sv[kc8 * 8 + 2 * q2] - m_ref));
          asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p1) : "f"(sv[kc8 * 8 + 2 * q2 + 1] - m_ref));
          if (m_ref == -INFINITY) p0 = p1 = 0.f;                       // -inf - -inf: nothing visible yet
          add += p0 + p1;
          const __half2 h = __floats2half2_rn(p0, p1);
          pk[q2] = *reinterpret_cast<const unsigned*>(&h);
        }
        *reinterpret_cast<uint4*>(pd + ((size_t)(4 * hf + kc8) * 128 + m) * 16) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
      }
      lsum += add;
      umma::fence_async_smem();
      umma::fence_before_sync();
      __syncwarp();
      if (l == 0) fl_mbar_arrive(&pFull[s]);
    }
    // ---------------------------------------------------------------- epilogue: each warp of a pair writes half of the channels
    float* half_sum = &half_max[n & 1][0][0];                           // the buffer the last step did not use
    if (hf == 1) half_sum[m] = lsum;
    pair_sync();
    if (hf == 0) { lsum += half_sum[m]; half_sum[128 + m] = lsum; }
    pair_sync();
    lsum = half_sum[128 + m];
    if (n > 0) warp_wait(&pvDone[(n - 1) % kFlStages], ((n - 1) / kFlStages) & 1);
    umma::fence_after_sync();
    if (P.partials) {                                                   // the tile is split: leave (m, l, acc) of this share
      float* rec = P.partials + (((size_t)blockIdx.z * a.R + row0 + r) * P.Hq + g * gqa + hq) * CR_QSA_PART;
      if (rowok && hf == 0) *reinterpret_cast<float2*>(rec) = make_float2(m_ref * 0.6931471805599453f, lsum);
#pragma unroll 1
      for (int c8 = 4 * hf; c8 < 4 * hf + 4; ++c8) {
        float o[32];
        umma::tmem_ld32(umma::tmem_addr(tm, w, kColO + 32 * c8), o);
        if (!rowok) continue;
#pragma unroll
        for (int c = 0; c < 32; c += 2) *reinterpret_cast<float2*>(rec + 2 + 32 * c8 + c) = n > 0 ? make_float2(o[c], o[c + 1]) : make_float2(0.f, 0.f);
      }
    }
    const bool ok = !P.partials && rowok && lsum > 0.f && !dead;
    const float inv = ok ? 1.f / lsum : 0.f;
    const int gr = row0 + r, h = g * gqa + hq;
    const size_t W = (size_t)P.Hq * 256;
    const float* gate = a.q + ((size_t)gr * P.Hq + h) * 512 + 256;
#pragma unroll 1
    for (int c8 = 4 * hf; c8 < 4 * hf + 4 && !P.partials; ++c8) {
      float o[32];
      umma::tmem_ld32(umma::tmem_addr(tm, w, kColO + 32 * c8), o);     // warp-collective: every lane takes part
      if (!ok) continue;
#pragma unroll
      for (int c = 0; c < 32; ++c) o[c] *= inv;
      if (a.context) {
        float4* cx = reinterpret_cast<float4*>(a.context + ((size_t)gr * P.Hq + h) * 256 + 32 * c8);
#pragma unroll
        for (int c = 0; c < 8; ++c) cx[c] = make_float4(o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
      }
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float4 gv = *reinterpret_cast<const float4*>(gate + 32 * c8 + 4 * c);
        o[4 * c] *= sigmoidf_(gv.x); o[4 * c + 1] *= sigmoidf_(gv.y); o[4 * c + 2] *= sigmoidf_(gv.z); o[4 * c + 3] *= sigmoidf_(gv.w);
      }
      const size_t at = (size_t)gr * W + h * 256 + 32 * c8;
      if (P.gated) {
        float4* dst = reinterpret_cast<float4*>(P.gated + at);
#pragma unroll
        for (int c = 0; c < 8; ++c) dst[c] = make_float4(o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
      } else if (P.fmt == CR_OUT_RAW_F32) {
        float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + at);
#pragma unroll
        for (int c = 0; c < 8; ++c) dst[c] = make_float4(o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
      } else {
        uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.out) + at);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          unsigned pk[4];
#pragma unroll
          for (int q2 = 0; q2 < 4; ++q2) {
            const __nv_bfloat162 b2 = __floats2bfloat162_rn(o[8 * c + 2 * q2], o[8 * c + 2 * q2 + 1]);
            pk[q2] = *reinterpret_cast<const unsigned*>(&b2);
          }
          dst[c] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        }
      }
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (w == kFlIssuer) umma::tmem_dealloc(tm, 512);
}

// The reference's out-projection input from gated fp32 rows: fp16(WHT128(RoundH(RoundH(o) * suh)) / sqrt(128))
// (engine/layers/qsa_long.h:476-489).  grid (Hq, R), 64 threads: a warp per 128-channel group.
__global__ void __launch_bounds__(64) qsa_out_transform_kernel(cr_qsa_args a, const float* gated, int Hq, const int* tile_count, int RT, int flash_max) {
  const int h = blockIdx.x, r = blockIdx.y, half = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (tile_count[r / RT] > flash_max) return;             // a row of the row-wise kernels, which transform their own output
  const int W = Hq * 256, c0 = h * 256 + half * 128 + lane * 4;
  const float4 o = *reinterpret_cast<const float4*>(gated + (size_t)r * W + c0);
  const __half* suh = reinterpret_cast<const __half*>(a.suh_o) + c0;
  float v[4] = {round_h(round_h(o.x) * __half2float(suh[0])), round_h(round_h(o.y) * __half2float(suh[1])),
                round_h(round_h(o.z) * __half2float(suh[2])), round_h(round_h(o.w) * __half2float(suh[3]))};
  wht128(v);
  __half* dst = reinterpret_cast<__half*>(a.out);
#pragma unroll
  for (int i = 0; i < 4; ++i) dst[out_index(r, c0 + i, W, a.pack_rows, a.pack_off)] = __float2half(v[i] * kHadNorm);
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

// Attention of the rows of `a` over the union lists; `gated` (rows x Hq x 256 floats) is needed for CR_OUT_EXL3_WHT.
cr_status qsa_flash_launch(const cr_geometry* g, const cr_qsa_args& a, const __half* q_hi, const int2* list, const int* count,
                           float* gated, float* partials, int splits, cr_out_format fmt, int flash_max, cudaStream_t stream) {
  static PerDeviceOnce configured;
  if (cr_status st = once_per_device(configured, [] {
        CR_CUDA(cudaFuncSetAttribute(qsa_flash_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFlashSmem));
        return CR_OK;
      })) return st;
  FlashParams P;
  P.a = a; P.q_hi = q_hi; P.list = list; P.count = count;
  P.RT = qsa_union_rows(g); P.cap = qsa_union_cap(P.RT);
  P.Hq = g->q_heads; P.Hkv = g->kv_heads; P.fmt = (int)fmt;
  P.gated = fmt == CR_OUT_EXL3_WHT && splits == 1 ? gated : nullptr;
  P.partials = splits > 1 ? partials : nullptr;
  P.flash_max = flash_max;
  CR_REQUIRE(fmt != CR_OUT_EXL3_WHT || gated, "qsa flash: the EXL3 output needs the gated fp32 scratch");
  const int tiles = (a.R + P.RT - 1) / P.RT;
  use_stream(stream);
  qsa_flash_tc_kernel<<<dim3(tiles, g->kv_heads, splits), kFlThreads, kFlashSmem, stream>>>(P);
  CR_LAUNCH_CHECK("qsa_flash_tc_kernel");
  if (P.gated) {
    qsa_out_transform_kernel<<<dim3(g->q_heads, a.R), 64, 0, stream>>>(a, gated, g->q_heads, count, P.RT, flash_max);
    CR_LAUNCH_CHECK("qsa_out_transform_kernel");
  }
  return CR_OK;
}

}  // namespace cr

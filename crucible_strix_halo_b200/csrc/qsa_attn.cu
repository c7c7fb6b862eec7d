// QSA attention over the attended positions for sm_100a (decode, verify, and the row-wise prefill path): the job of
// QsaGqaSplitKernel and QsaMergeKernel (engine/layers/qsa_long.h:399-499) in one kernel.
//
// A unit is a (row, KV head): up to 513 entries (selected blocks of 4 positions, then the open block), walked by one or
// more streams.  A stream is one warp (two where the KV group has more than 8 query heads, half of the heads each) that
// takes 16 positions at a time, with the positions as the M rows and the query heads as the N = 8 columns of mma.sync
// m16n8k16, so no row of the product is padding:
//   S^T[16 x 8] = K[16 x 256] Q^T        Q stays in registers as column fragments
//   O^T[256 x 8] += V^T[256 x 16] P^T    V read transposed by ldmatrix; P turned by movmatrix, in registers
// K and V are fp16 in the cache.  Q and P are fp32 values: each is split into an fp16 head and an fp16 remainder and
// multiplied twice, which keeps the products at fp32 accuracy.  Every stream has a ring of three 8 KB halves (K or V of
// 16 positions, one 512-byte row per cp.async instruction, XOR-swizzled in 16-byte pieces) of which two are in flight
// while the third is multiplied, and nothing in the loop crosses warps: no block barrier, no shared maxima.
// Streams of a unit are merged by log-sum-exp in shared memory and, when a unit spans several CTAs, over a thread-block
// cluster through distributed shared memory; the sigmoid gate and the output transform follow in place, so no partial
// sum goes through HBM.
//
// Bound: the gather.  Random 512-byte rows of a 512 MB cache arrive at 8.5 TB/s (16 MB: 20 TB/s).  The form before this
// one (a CTA per (row, KV head, split), heads as M rows, Q re-read from shared memory for every tile, partials merged by
// a second kernel) was held by shared-memory reads and barriers: 2,048 rows at 262,144 positions took 1,875 us plus
// 180 us of merge, 700 us now (12 TB/s of gathers: the rows walk their ascending positions side by side, so the rows in
// flight share a region of the cache that L2 holds; from L2 alone 666 us, where every byte's way into and out of shared
// memory takes three quarters of its bandwidth); 72 verify rows at 131,072 105 + 12 us, 53 us now.
// Steps of few rows are a chain of round trips (parameters, selection, K, V, merge over the CTA, over the cluster): 10.8 us for a
// row at 1,501 positions, 13 for four at 262,144, 16.4 for four of 24 heads at 32,003 while every warp fetched its query fragments
// itself (256 line look-ups each), the count of a selection came before its ids, gates were asked for at the end and the
// parts of a merge one by one; 8.3, 9.0 and 14.1 us now.
#include <climits>
#include <cooperative_groups.h>
#include "qsa.cuh"

namespace cg = cooperative_groups;

namespace cr {

constexpr int kTok = 16;                       // positions per tile: four blocks
constexpr int kHalfBytes = kTok * 512;         // K or V rows of a tile
constexpr int kSlots = 3;                      // halves in a stream's ring
constexpr int kRingBytes = kSlots * kHalfBytes;
constexpr int kAccLd = 260;                    // floats per head of an accumulator image in shared memory (conflict-free writes)
constexpr int kMaxWarps = 12;

// Streams of a CTA by head groups: 8 of one warp, or 6 of two (168 registers a thread fill the register file).
template <int NG> constexpr int kStreams = NG == 1 ? 8 : 6;
template <int NG> constexpr int kAttnThreads = kStreams<NG> * NG * 32;
template <int NG> constexpr size_t kAttnSmem = (size_t)kStreams<NG> * kRingBytes;

struct AttnShape {
  int spu;                                     // streams of a CTA that share a unit; kStreams / spu units per CTA
  int cluster;                                 // CTAs per unit (spu = all streams then)
};

__device__ __forceinline__ void attn_cp16(unsigned dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src));
}
__device__ __forceinline__ void attn_cp16_or_zero(unsigned dst, const void* src, bool valid) {
  const int bytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void ldsm_x4(unsigned (&r)[4], unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(unsigned (&r)[4], unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ unsigned transpose8(unsigned x) {   // 8 x 8 fp16 of a warp: row g, columns 2 tq, 2 tq + 1 per lane
  unsigned y;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(y) : "r"(x));
  return y;
}
__device__ __forceinline__ void mma_f16(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void split2(float x, float y, unsigned& hi, unsigned& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 b = __half22float2(h);
  const __half2 r = __floats2half2_rn(x - b.x, y - b.y);
  hi = *reinterpret_cast<const unsigned*>(&h);
  lo = *reinterpret_cast<const unsigned*>(&r);
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// grid (cluster x ceil(Rmax * Hkv / units per CTA), 1, spans).  HKV: the cache's KV heads where they are two (row pitches
// become constants), else 0.
// UNIT: a CTA, or a cluster of them, has one unit (steps); without it streams have units of their own (long parts).  Two kernels: what
// the one form needs on its way from the selection to the output costs the other's loop 1 to 2 % in registers and instructions.
template <int NG, int HKV, bool UNIT>
__global__ void __launch_bounds__(kAttnThreads<NG>, 1) qsa_attn_kernel(const __grid_constant__ QsaParams P, const AttnShape shape, float* partials,
                                                                       int p0, int p1, int fmt) {
  extern __shared__ __align__(1024) unsigned char ring_raw[];
  __shared__ float ml_s[kMaxWarps][8][2];              // (m, l) of every stream's heads
  __shared__ float2 cta_ml[16];                        // (m, l) of the CTA's merged unit, read by the cluster
  pdl_release();
  constexpr int W = kStreams<NG>;
  const cr_qsa_args& a = P.span[blockIdx.z];
  touch_params(a);
  pdl_wait();
  const int t = threadIdx.x, warp = t >> 5, l = t & 31, g8 = l >> 2, tq = l & 3;
  const int stream = warp / NG, hg = warp % NG;
  const int upc = UNIT ? 1 : W / shape.spu, crank = UNIT && shape.cluster > 1 ? (int)(blockIdx.x % shape.cluster) : 0;
  const int unit = UNIT ? (int)(blockIdx.x / shape.cluster) : (int)blockIdx.x * upc + stream / shape.spu, sub = UNIT ? stream : stream % shape.spu;
  const int r = unit / P.Hkv, g = unit % P.Hkv;
  const int gqa = P.Hq / P.Hkv, gh = (gqa + NG - 1) / NG;           // heads of a head group
  const int heads = min(gh, gqa - hg * gh);
  // Units past the rows, and rows of the tiled kernel: with one unit per CTA or cluster everybody leaves, else the stream idles
  // through the CTA's barriers.
  const bool live = r < a.R && !qsa_row_is_tiled(P, r);
  if (upc == 1 && !live) return;

  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
  float O[16][4];
#pragma unroll
  for (int i = 0; i < 16; ++i) O[i][0] = O[i][1] = O[i][2] = O[i][3] = 0.f;
  unsigned char* ring = ring_raw + (size_t)stream * kRingBytes;

  if (live) {
    const int p = a.pos0 + r, nb = (p + 1) / 4;
    const int* sel = a.sel + (size_t)r * CR_SEL_BLOCKS;
    // Where the CTA has one unit its query heads come in once, beside the selection: [head][256] with the 32-byte pieces of a row
    // XORed by the head, so that the fragment reads meet no bank twice.  (Every warp loading them as fragments cost 256 line
    // look-ups a warp: 2 us of a step's 9 to 16.)
    float* qs = reinterpret_cast<float*>(ring_raw + (size_t)W * kRingBytes);
    const bool q_shared = UNIT && ((uintptr_t)a.q & 15) == 0;    // a rank's partials read no gates: its rows may lie at 8 bytes
    if (q_shared) {
      const float* q = a.q + ((size_t)r * P.Hq + g * gqa) * 512;
      for (int i = t; i < gqa * 64; i += kAttnThreads<NG>) {
        const int hd = i >> 6, pc = i & 63;
        attn_cp16((unsigned)__cvta_generic_to_shared(qs) + hd * 1024 + (pc ^ ((hd & 7) << 1)) * 16, q + (size_t)hd * 512 + pc * 4);
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    // The selection holds all or 512 blocks, as the row's length says: its ids are asked for in that belief, beside the count.
    const int counted = __ldcg(a.nsel + r);
    int ns = nb <= CR_SEL_BLOCKS ? -1 : CR_SEL_BLOCKS;
    int full, e_hi, e0, tiles, ids, ids_next;
    auto load_ids = [&](int k) {                           // lane l: entry e0 + 32 k + l of this stream
      const int e = e0 + 32 * k + l;
      return e < e_hi ? (ns < 0 || e >= full ? (e >= full ? nb : e) : sel[e]) : -1;
    };
    for (;; ns = counted) {
      // Entries: the selected blocks (all complete blocks when dense), then the open block.  They ascend, so those that reach
      // into a rank's window [p0, p1) are one contiguous range.
      full = ns < 0 ? nb : ns;
      int e_lo = 0;
      e_hi = full + ((p + 1) % 4 != 0 ? 1 : 0);
      if (p0 > 0 || p1 <= p) {
        auto entry_at_least = [&](int blk) {               // first entry whose block is >= blk
          if (ns < 0) return min(blk, e_hi);
          int lo = 0, hi = full;
          while (lo < hi) { const int mid = (lo + hi) >> 1; if (sel[mid] < blk) lo = mid + 1; else hi = mid; }
          return lo == full && nb < blk ? e_hi : lo;
        };
        const int lo = entry_at_least(p0 / 4), hi = p1 > p ? e_hi : entry_at_least((p1 + 3) / 4);
        e_lo = lo; e_hi = min(hi, e_hi);
      }
      const int tiles_all = max(e_hi - e_lo + 3, 0) / 4, streams = shape.spu * shape.cluster, s_idx = crank * shape.spu + sub;
      const int tb = tiles_all / streams, trem = tiles_all % streams;
      tiles = tb + (s_idx < trem ? 1 : 0);
      e0 = e_lo + 4 * (s_idx * tb + min(s_idx, trem));     // first entry of this stream
      // Block ids: lane l of `ids` holds entry e0 + 32 k + l of the current group of eight tiles, `ids_next` the next group.
      ids = load_ids(0); ids_next = load_ids(1);
      if (counted == ns) break;
    }
    const size_t row_bytes = HKV ? (size_t)HKV * 512 : (size_t)P.Hkv * 512;
    const char* kc = reinterpret_cast<const char*>(a.c.k) + (size_t)g * 512 + l * 16;
    const char* vc = reinterpret_cast<const char*>(a.c.v) + (size_t)g * 512 + l * 16;
    const unsigned ring_s = (unsigned)__cvta_generic_to_shared(ring), ring_l = ring_s + l * 16;
    const int lo_pos = max(p0, 0), hi_pos = min(p, p1 - 1);          // visible positions
    // Tiles before this one (of the stream's) hold complete selected blocks inside the window: nothing to mask.
    const int whole_tiles = p0 <= 0 && p1 > p ? (full - e0) >> 2 : 0;
    int blk[4];                                          // blocks of the tile whose K half was issued last
    auto issue = [&](const char* base, int half, bool whole) {       // the 16 rows of the tile in blk, into slot half % kSlots
      const unsigned slot = ring_l + (half % kSlots) * kHalfBytes;    // slots are 512-byte aligned: the swizzle is one XOR
#pragma unroll
      for (int i4 = 0; i4 < kTok / 4 / NG; ++i4) {
        const int b = NG == 1 ? blk[i4] : (hg == 0 ? blk[i4] : blk[2 + i4]);
        const char* src = base + (size_t)(unsigned)b * (4 * row_bytes);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int kk = 4 * i4 + i;                     // row of this warp's share: 8 hg + kk where two warps share a stream
          const unsigned dst = (slot ^ ((kk & 7) << 4)) + (NG == 1 ? kk : 8 * hg + kk) * 512;
          if (whole) {
            attn_cp16(dst, src + i * row_bytes);
          } else {
            const int pos = 4 * b + i;
            const bool ok = b >= 0 && pos >= lo_pos && pos <= hi_pos;
            attn_cp16_or_zero(dst, ok ? src + i * row_bytes : base, ok);
          }
        }
      }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;\n" ::: "memory"); };
    auto visible = [&](bool whole) {                     // bit k: position k of the tile in blk is attended
      if (whole) return 0xFFFFu;
      const int b = l < kTok ? (l < 8 ? (l < 4 ? blk[0] : blk[1]) : (l < 12 ? blk[2] : blk[3])) : -1;
      const int pos = 4 * b + (l & 3);
      return __ballot_sync(0xffffffffu, b >= 0 && pos >= lo_pos && pos <= hi_pos);
    };
    auto take_blocks = [&](int tile) {                   // tile's four block ids (called for tile = 0, 1, 2, ...)
      if ((tile & 7) == 0 && tile > 0) { ids = ids_next; ids_next = load_ids((tile >> 3) + 1); }
#pragma unroll
      for (int j = 0; j < 4; ++j) blk[j] = __shfl_sync(0xffffffffu, ids, 4 * (tile & 7) + j);
    };
    auto pair_sync = [&] {                               // the warps of a stream
      if constexpr (NG == 1) __syncwarp();
      else asm volatile("bar.sync %0, 64;\n" ::"r"(1 + stream) : "memory");
    };
    unsigned see = 0, see_next = 0;
    if (tiles > 0) { take_blocks(0); see = visible(0 < whole_tiles); issue(kc, 0, 0 < whole_tiles); }
    commit();
    if (tiles > 0) issue(vc, 1, 0 < whole_tiles);
    commit();
    if (tiles > 1) { take_blocks(1); see_next = visible(1 < whole_tiles); issue(kc, 2, 1 < whole_tiles); }
    commit();
    // Query heads of the group as column fragments, fp16 head and remainder, while the first halves are in flight.
    unsigned qh[16][2], ql[16][2];
    {
      const bool have = g8 < heads;
      const int hd = hg * gh + min(g8, heads - 1);
      auto take = [&](int ks, int j, float2 v) {
        if (!have) v = make_float2(0.f, 0.f);
        split2(v.x, v.y, qh[ks][j], ql[ks][j]);
      };
      if (q_shared) {
        asm volatile("cp.async.wait_group 3;\n" ::: "memory");
        __syncthreads();
        const float* q = qs + hd * 256 + 2 * tq;
#pragma unroll
        for (int ks = 0; ks < 16; ++ks)
#pragma unroll
          for (int j = 0; j < 2; ++j) take(ks, j, *reinterpret_cast<const float2*>(q + ((2 * ks + j) ^ (hd & 7)) * 8));
      } else {
        const float* q = a.q + ((size_t)r * P.Hq + g * gqa + hd) * 512 + 2 * tq;
#pragma unroll
        for (int ks = 0; ks < 16; ++ks)
#pragma unroll
          for (int j = 0; j < 2; ++j) take(ks, j, *reinterpret_cast<const float2*>(q + (2 * ks + j) * 8));
      }
    }
    constexpr float kScale = 0.0625f * 1.4426950408889634f;           // logits / 16, in powers of two
    // this lane's ldmatrix rows: K: matrices (positions 0-7 | 8-15) x (first | second 8 channels); V: the transpose of that
    const int mi = l >> 3, k_row = (l & 7) + (mi & 1) * 8, v_row = (l & 7) + (mi >> 1) * 8;
    const unsigned k_addr = k_row * 512 + (((mi >> 1) ^ (l & 7)) << 4), v_addr = v_row * 512 + (((mi & 1) ^ (l & 7)) << 4);   // ^ 32 per 16 channels
    for (int i = 0; i < tiles; ++i) {
      asm volatile("cp.async.wait_group 2;\n" ::: "memory");
      pair_sync();
      const unsigned ks_base = ring_s + ((2 * i) % kSlots) * kHalfBytes + k_addr;
      float s[4] = {0.f, 0.f, 0.f, 0.f}, s2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int ks = 0; ks < 16; ++ks) {
        unsigned ka[4];
        ldsm_x4(ka, ks_base ^ (ks << 5));
        mma_f16(s, ka, qh[ks][0], qh[ks][1]);
        mma_f16(s2, ka, ql[ks][0], ql[ks][1]);
      }
      pair_sync();                                       // the K half is free
      if (i + 1 < tiles) issue(vc, 2 * i + 3, i + 1 < whole_tiles);   // blk still holds tile i + 1
      commit();
      const bool v0 = (see >> g8) & 1u, v1 = (see >> (g8 + 8)) & 1u;
#pragma unroll
      for (int j = 0; j < 4; ++j) s[j] = (j < 2 ? v0 : v1) ? (s[j] + s2[j]) * kScale : -INFINITY;
      float mx[2] = {fmaxf(s[0], s[2]), fmaxf(s[1], s[3])};
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {
        mx[0] = fmaxf(mx[0], __shfl_xor_sync(0xffffffffu, mx[0], o));
        mx[1] = fmaxf(mx[1], __shfl_xor_sync(0xffffffffu, mx[1], o));
      }
      // The reference maximum moves only when a logit exceeds it by more than 2^8: O is rescaled once or twice per stream, and
      // probabilities up to 256 lose nothing in their fp16 head and remainder.
      if (__any_sync(0xffffffffu, mx[0] > m_run[0] + 8.f || mx[1] > m_run[1] + 8.f)) {
        float corr[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float mn = fmaxf(m_run[j], mx[j]);
          corr[j] = m_run[j] > -INFINITY ? ex2(m_run[j] - mn) : 0.f;
          l_run[j] *= corr[j];
          m_run[j] = mn;
        }
#pragma unroll
        for (int mt = 0; mt < 16; ++mt) { O[mt][0] *= corr[0]; O[mt][1] *= corr[1]; O[mt][2] *= corr[0]; O[mt][3] *= corr[1]; }
      }
      float e[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) e[j] = s[j] > -INFINITY ? ex2(s[j] - m_run[j & 1]) : 0.f;
      l_run[0] += e[0] + e[2];
      l_run[1] += e[1] + e[3];
      unsigned ph[2], pl[2];
      split2(e[0], e[1], ph[0], pl[0]);
      split2(e[2], e[3], ph[1], pl[1]);
#pragma unroll
      for (int j = 0; j < 2; ++j) { ph[j] = transpose8(ph[j]); pl[j] = transpose8(pl[j]); }
      asm volatile("cp.async.wait_group 2;\n" ::: "memory");
      pair_sync();
      const unsigned vs_base = ring_s + ((2 * i + 1) % kSlots) * kHalfBytes + v_addr;
#pragma unroll
      for (int mt = 0; mt < 16; ++mt) {
        unsigned va[4];
        ldsm_x4_trans(va, vs_base ^ (mt << 5));
        mma_f16(O[mt], va, ph[0], ph[1]);
        mma_f16(O[mt], va, pl[0], pl[1]);
      }
      pair_sync();                                       // the V half is free
      see = see_next;
      if (i + 2 < tiles) { take_blocks(i + 2); see_next = visible(i + 2 < whole_tiles); issue(kc, 2 * i + 4, i + 2 < whole_tiles); }
      commit();
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      l_run[0] += __shfl_xor_sync(0xffffffffu, l_run[0], o);
      l_run[1] += __shfl_xor_sync(0xffffffffu, l_run[1], o);
    }
  }

  // ---- merge: every stream leaves its accumulator as [head][channel] in its ring, (m, l) beside it
  float* acc = reinterpret_cast<float*>(ring) + (size_t)hg * 8 * kAccLd;
  if (NG == 2) asm volatile("bar.sync %0, 64;\n" ::"r"(1 + stream) : "memory");   // the other warp of the stream has left the ring
  else __syncwarp();
#pragma unroll
  for (int mt = 0; mt < 16; ++mt) {
    float* d = acc + 2 * tq * kAccLd + 16 * mt + g8;
    d[0] = O[mt][0]; d[kAccLd] = O[mt][1]; d[8] = O[mt][2]; d[kAccLd + 8] = O[mt][3];
  }
  if (g8 == 0) {
    ml_s[warp][2 * tq][0] = m_run[0]; ml_s[warp][2 * tq][1] = l_run[0];
    ml_s[warp][2 * tq + 1][0] = m_run[1]; ml_s[warp][2 * tq + 1][1] = l_run[1];
  }
  if (shape.spu == 1) {
    if (NG == 1) __syncwarp();
    else asm volatile("bar.sync %0, 64;\n" ::"r"(1 + stream) : "memory");
  } else {
    __syncthreads();
  }
  if ((!UNIT || shape.cluster == 1) && !live) return;
  // This CTA's merged (m, l, acc) of head hd, channels c .. c + 3.  (One part at a time and the gate at the end: long parts, where a
  // stream has its unit to itself, lose 1.5 % to eight parts or the gate in flight.)
  const int first_stream = stream - sub;
  auto merged = [&](int hd, int c, float& m, float& lsum) {
    const int hg_ = hd / gh, hl = hd % gh;
    m = -INFINITY;
    for (int s = 0; s < shape.spu; ++s) m = fmaxf(m, ml_s[(first_stream + s) * NG + hg_][hl][0]);
    lsum = 0.f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < shape.spu; ++s) {
      const float ms = ml_s[(first_stream + s) * NG + hg_][hl][0], f = ms > -INFINITY ? ex2(ms - m) : 0.f;
      lsum = fmaf(ml_s[(first_stream + s) * NG + hg_][hl][1], f, lsum);
      const float4 x = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(ring_raw + (size_t)(first_stream + s) * kRingBytes) + (size_t)(hg_ * 8 + hl) * kAccLd + c);
      o.x = fmaf(x.x, f, o.x); o.y = fmaf(x.y, f, o.y); o.z = fmaf(x.z, f, o.z); o.w = fmaf(x.w, f, o.w);
    }
    return o;
  };
  auto gate_of = [&](int hd, int c) {
    return partials ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4*>(a.q + ((size_t)r * P.Hq + g * gqa + hd) * 512 + 256 + c);
  };
  auto finish = [&](int hd, int c, float m, float lsum, float4 o, float4 gate) {
    const int h = g * gqa + hd;
    if (partials) {                                      // a rank's partial: (m, l, acc) with m as a natural logarithm
      float* dst = partials + ((size_t)(P.base[blockIdx.z] + r) * P.Hq + h) * CR_QSA_PART;
      if (c == 0) { dst[0] = m * 0.6931471805599453f; dst[1] = lsum; }
      *reinterpret_cast<float2*>(dst + 2 + c) = make_float2(o.x, o.y);
      *reinterpret_cast<float2*>(dst + 4 + c) = make_float2(o.z, o.w);
      return;
    }
    const float inv = 1.f / lsum;
    emit_group(a, P.Hq, r, h, c, make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv), gate, fmt);
  };
  const int uw = sub * NG + hg, uwarps = shape.spu * NG;               // this warp among the warps of its unit in this CTA
  if (!UNIT || shape.cluster == 1) {
    for (int gi = uw; gi < 2 * gqa; gi += uwarps) {                     // groups: (head, 128 channels)
      float m, lsum;
      const int hd = gi >> 1, c = (gi & 1) * 128 + 4 * l;
      const float4 o = merged(hd, c, m, lsum);
      finish(hd, c, m, lsum, o, gate_of(hd, c));
    }
    return;
  }
  if constexpr (UNIT) {
  // (m, l) of `n` parts (at most 8), lane k & 7 holding those of part k: the factor of that part's accumulator; m and l become those of
  // the whole.
  auto weigh = [&](int n, float& m, float& lsum) {
    const bool have = (l & 7) < n;
    const float mk = have ? m : -INFINITY;
    m = mk;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float f = mk > -INFINITY ? ex2(mk - m) : 0.f;
    lsum = have ? lsum * f : 0.f;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    return f;
  };
  auto weighted = [&](const float4 (&x)[8], int n, float f) {
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float fk = __shfl_sync(0xffffffffu, f, k);
      if (k < n) { o.x = fmaf(x[k].x, fk, o.x); o.y = fmaf(x[k].y, fk, o.y); o.z = fmaf(x[k].z, fk, o.z); o.w = fmaf(x[k].w, fk, o.w); }
    }
    return o;
  };
  // cluster: the CTA's merged unit goes to shared memory behind the ring images of the first stream, then every CTA takes a
  // share of the groups over all CTAs: at most one group per warp (two CTAs have 16 or 24 warps, as many as there are groups)
  cg::cluster_group cluster = cg::this_cluster();
  float* mine = reinterpret_cast<float*>(ring_raw + (size_t)W * kRingBytes);
  const int gi_out = crank + shape.cluster * warp, hd_out = gi_out >> 1, c_out = (gi_out & 1) * 128 + 4 * l;
  const bool emits = gi_out < 2 * gqa;
  float4 gate = make_float4(0.f, 0.f, 0.f, 0.f);
  if (emits) gate = gate_of(hd_out, c_out);                           // in flight through the merge
  for (int hd = warp; hd < gqa; hd += W * NG) {                        // a head per warp: both halves share their weights
    const int hg_ = hd / gh, hl = hd % gh;
    const float* img = reinterpret_cast<const float*>(ring_raw) + (size_t)(hg_ * 8 + hl) * kAccLd + 4 * l;
    float4 x[2][8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < W) {
        x[0][k] = *reinterpret_cast<const float4*>(img + (size_t)k * (kRingBytes / 4));
        x[1][k] = *reinterpret_cast<const float4*>(img + (size_t)k * (kRingBytes / 4) + 128);
      }
    const float* ml = ml_s[min(l & 7, W - 1) * NG + hg_][hl];
    float m = ml[0], lsum = ml[1];
    const float f = weigh(W, m, lsum);
    *reinterpret_cast<float4*>(mine + hd * 256 + 4 * l) = weighted(x[0], W, f);
    *reinterpret_cast<float4*>(mine + hd * 256 + 128 + 4 * l) = weighted(x[1], W, f);
    if (l == 0) cta_ml[hd] = make_float2(m, lsum);
  }
  cluster.sync();
  float m = -INFINITY, lsum = 0.f;
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  if (emits) {
    float4 x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < shape.cluster) x[k] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(mine, k) + hd_out * 256 + c_out);
    const float2 ml = cluster.map_shared_rank(&cta_ml[0], min(l & 7, shape.cluster - 1))[hd_out];
    m = ml.x; lsum = ml.y;
    const float f = weigh(shape.cluster, m, lsum);
    o = weighted(x, shape.cluster, f);
  }
  cluster.barrier_arrive();                              // this CTA has read the others' images
  if (emits) finish(hd_out, c_out, m, lsum, o, gate);
  cluster.barrier_wait();                                // the own images stay until every CTA has read them
  }
}

// Merge of the partial records of several ranks or of a tile's splits (QsaMergeKernel, engine/layers/qsa_long.h:458-499), gate and output
// transform.  grid (Hq, R), 64 threads: a warp per 128-channel group.  Record p of (row, head) lies at
// partials[((p * rows + row) * Hq + h) * 258].
__global__ void __launch_bounds__(64) qsa_merge_kernel(const __grid_constant__ QsaParams P, const float* partials, int nparts, int fmt) {
  pdl_release();
  pdl_wait();
  const cr_qsa_args& a = P.span[0];
  const int h = blockIdx.x, r = blockIdx.y, l = threadIdx.x & 31, c = (threadIdx.x >> 5) * 128 + 4 * l;
  if (P.tile_count && !qsa_row_is_tiled(P, r)) return;   // a row of the row-wise kernel
  auto rec = [&](int p) { return partials + (((size_t)p * a.R + r) * P.Hq + h) * CR_QSA_PART; };
  float pm = -INFINITY, pl = 0.f;                        // lane p: (m, l) of record p
  if (l < nparts) {
    const float2 v = *reinterpret_cast<const float2*>(rec(l));
    pl = v.y;
    pm = pl != 0.f ? v.x : -INFINITY;
  }
  const float mx = warp_max(pm);
  const float f = pl != 0.f ? __expf(pm - mx) : 0.f;
  const float lsum = warp_sum(pl * f);
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int p = 0; p < nparts; ++p) {
    const float fp = __shfl_sync(0xffffffffu, f, p);
    const float2 x = *reinterpret_cast<const float2*>(rec(p) + 2 + c), y = *reinterpret_cast<const float2*>(rec(p) + 4 + c);
    o.x = fmaf(x.x, fp, o.x); o.y = fmaf(x.y, fp, o.y); o.z = fmaf(y.x, fp, o.z); o.w = fmaf(y.y, fp, o.w);
  }
  const float4 gate = *reinterpret_cast<const float4*>(a.q + ((size_t)r * P.Hq + h) * 512 + 256 + c);
  const float inv = 1.f / lsum;
  emit_group(a, P.Hq, r, h, c, make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv), gate, fmt);
}

// Streams of a unit.  The pass holds `fits[k]` clusters of 2^k CTAs at a time (an SM each); with s streams per unit it takes
// that many waves of (longest unit's tiles / s + the set-up and merge of a stream, worth about four tiles).
// One stream per unit is the cheapest form but leaves SMs idle when units are few and ends in a ragged wave when they
// are not many; a cluster (s above one CTA's streams) pays only while SMs would idle otherwise.  A cluster lies in one
// group of SMs, so that fewer fit than the SMs would hold (15 of eight CTAs where 148 SMs count 18), and one cluster too many doubles
// the time of a step: 16 units (eight sessions of one row) 18.5 us of 16 heads and 26.6 of 24 by the count of SMs, 12.5 and 20.6 by
// what fits; 36 units 23.7 and 40.2, now 17.8 and 32.8.
static AttnShape attn_shape(int streams, long long units, int tiles, const int (&fits)[4]) {
  AttnShape best{1, 1};
  double best_cost = 1e30;
  for (int spu = 1; spu <= streams; ++spu) {
    if (streams % spu) continue;
    for (int k = 0; k < 4; ++k) {
      const int cl = 1 << k;
      if (cl > 1 && (spu != streams || units > fits[k])) break;
      if (spu * cl > 1 && spu * cl > tiles) break;
      const long long clusters = cl > 1 ? units : (units * spu + streams - 1) / streams;
      const long long waves = (clusters + fits[k] - 1) / fits[k];
      const double cost = (double)waves * ((tiles + spu * cl - 1) / (spu * cl) + 4);
      if (cost < best_cost - 1e-9) { best_cost = cost; best = AttnShape{spu, cl}; }
    }
  }
  return best;
}

template <int NG, int HKV>
static cr_status attn_launch_t(const QsaParams& P, int Rmax, int n, long long units, int tiles, float* partials, int p0, int p1, int fmt, cudaStream_t stream) {
  static PerDeviceOnce configured;
  static int fits_on[64][4];                            // per device: clusters of 1, 2, 4 and 8 CTAs that run at once
  constexpr size_t smem = kAttnSmem<NG> + 12 * 256 * sizeof(float);   // + the query heads of a CTA's unit, then its merged unit
  int dev = 0;
  CR_CUDA(cudaGetDevice(&dev));
  dev &= 63;
  if (cr_status st = once_per_device(configured, [dev] {
        CR_CUDA(cudaFuncSetAttribute(qsa_attn_kernel<NG, HKV, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        CR_CUDA(cudaFuncSetAttribute(qsa_attn_kernel<NG, HKV, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        fits_on[dev][0] = sm_count();
        for (int k = 1; k < 4; ++k) {
          cudaLaunchConfig_t cfg = {};
          cfg.gridDim = dim3(sm_count() >> k << k); cfg.blockDim = dim3(kAttnThreads<NG>); cfg.dynamicSmemBytes = smem;
          cudaLaunchAttribute attr;
          attr.id = cudaLaunchAttributeClusterDimension;
          attr.val.clusterDim.x = 1 << k; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
          cfg.attrs = &attr; cfg.numAttrs = 1;
          CR_CUDA(cudaOccupancyMaxActiveClusters(&fits_on[dev][k], qsa_attn_kernel<NG, HKV, true>, &cfg));
        }
        return CR_OK;
      })) return st;
  const AttnShape shape = attn_shape(kStreams<NG>, units, tiles, fits_on[dev]);
  const int upc = kStreams<NG> / shape.spu;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(shape.cluster * ((Rmax * P.Hkv + upc - 1) / upc), 1, n);
  cfg.blockDim = dim3(kAttnThreads<NG>);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (pdl_enabled()) { attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[na++].val.programmaticStreamSerializationAllowed = 1; }
  if (shape.cluster > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = shape.cluster; attr[na].val.clusterDim.y = 1; attr[na++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr; cfg.numAttrs = na;
  CR_CUDA(cudaLaunchKernelEx(&cfg, upc == 1 ? qsa_attn_kernel<NG, HKV, true> : qsa_attn_kernel<NG, HKV, false>, P, shape, partials, p0, p1, fmt));
  CR_LAUNCH_CHECK("qsa_attn_kernel");
  return CR_OK;
}

cr_status qsa_attn_launch(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, float* partials, int p0, int p1, cr_out_format fmt,
                          cudaStream_t stream, const QsaTileSplit* tiles) {
  use_stream(stream);
  int row_base = 0;
  for (int s0 = 0; s0 < n_spans; s0 += kMaxSpans) {
    const int n = n_spans - s0 < kMaxSpans ? n_spans - s0 : kMaxSpans;
    QsaParams P;
    qsa_fill_params(P, g, spans + s0, n);
    if (tiles) { P.tile_count = tiles->count; P.tile_rows = tiles->rows; P.tile_max = tiles->max; P.tile_mixed = tiles->mixed; }
    long long units = 0;
    int last = 0;                                        // newest position of any row
    for (int s = 0; s < n; ++s) {
      P.base[s] += row_base;
      units += (long long)spans[s0 + s].R * g->kv_heads;
      last = max(last, spans[s0 + s].pos0 + spans[s0 + s].R - 1);
    }
    const int most = (min(last / 4 + 1, CR_SEL_BLOCKS + 1) + 3) / 4, Rmax = qsa_max_rows(spans + s0, n);
    const bool one = g->q_heads / g->kv_heads <= 8, two_kv = g->kv_heads == 2;
    auto launch = one ? (two_kv ? attn_launch_t<1, 2> : attn_launch_t<1, 0>) : (two_kv ? attn_launch_t<2, 2> : attn_launch_t<2, 0>);
    const cr_status st = launch(P, Rmax, n, units, most, partials, p0, p1, (int)fmt, stream);
    if (st) return st;
    for (int s = 0; s < n; ++s) row_base += spans[s0 + s].R;
  }
  return CR_OK;
}

cr_status qsa_merge_launch(const cr_geometry* g, const cr_qsa_args& a, int nparts, const float* partials, cr_out_format fmt, cudaStream_t stream,
                           const QsaTileSplit* tiles) {
  QsaParams P;
  qsa_fill_params(P, g, &a, 1);
  if (tiles) { P.tile_count = tiles->count; P.tile_rows = tiles->rows; P.tile_max = tiles->max; P.tile_mixed = tiles->mixed; }
  use_stream(stream);
  CR_CUDA(launch_pdl(qsa_merge_kernel, dim3(g->q_heads, a.R), dim3(64), 0, stream, P, partials, nparts, (int)fmt));
  CR_LAUNCH_CHECK("qsa_merge_kernel");
  return CR_OK;
}

static cr_status check_out(const cr_qsa_args* spans, int n, cr_out_format fmt, const char* who) {
  CR_REQUIRE(fmt == CR_OUT_RAW_F32 || fmt == CR_OUT_RAW_BF16 || fmt == CR_OUT_EXL3_WHT, "%s: bad output format", who);
  for (int s = 0; s < n; ++s) {
    CR_REQUIRE(spans[s].out, "%s: span %d has no output buffer", who, s);
    CR_REQUIRE(fmt != CR_OUT_EXL3_WHT || spans[s].suh_o, "%s: span %d needs suh_o for the EXL3 output", who, s);
    CR_REQUIRE(fmt == CR_OUT_EXL3_WHT || spans[s].pack_rows == 0, "%s: packed layout only with the EXL3 output", who);
  }
  return CR_OK;
}

}  // namespace cr

// What the reference's callers size by; the entry points below ignore their scratch, the parts of a row being merged on chip.
extern "C" size_t cr_qsa_scratch_bytes(const cr_geometry* g, int rows) {
  if (!g || rows < 1) return 0;
  return (size_t)rows * g->q_heads * CR_QSA_SPLITS * CR_QSA_PART * sizeof(float);
}

extern "C" cr_status cr_qsa_attn(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, void*, size_t, cr_out_format fmt, void* stream) {
  using namespace cr;
  if (cr_status s = qsa_validate(g, spans, n_spans, CR_MAX_STEP_ROWS, "cr_qsa_attn")) return s;
  if (cr_status s = check_out(spans, n_spans, fmt, "cr_qsa_attn")) return s;
  return qsa_attn_launch(g, spans, n_spans, nullptr, 0, INT_MAX, fmt, (cudaStream_t)stream);
}

extern "C" cr_status cr_qsa_step(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, void*, size_t, cr_out_format fmt, void* stream) {
  using namespace cr;
  if (cr_status s = qsa_validate(g, spans, n_spans, CR_MAX_STEP_ROWS, "cr_qsa_step")) return s;
  if (cr_status s = check_out(spans, n_spans, fmt, "cr_qsa_step")) return s;
  cudaStream_t st = (cudaStream_t)stream;
  if (cr_status s = qsa_prep_launch(g, spans, n_spans, 0, nullptr, 0, st, false, true)) return s;
  if (cr_status s = qsa_select_launch(g, spans, n_spans, st, true)) return s;
  return qsa_attn_launch(g, spans, n_spans, nullptr, 0, INT_MAX, fmt, st);
}

extern "C" cr_status cr_qsa_shard_attn(const cr_geometry* g, const cr_qsa_args* a, int p0, int p1, float* partials, void*, size_t, void* stream) {
  using namespace cr;
  if (cr_status s = qsa_validate(g, a, 1, CR_MAX_PREFILL_ROWS, "cr_qsa_shard_attn", 0)) return s;
  CR_REQUIRE(partials && p0 >= 0 && p1 >= p0, "cr_qsa_shard_attn: bad position window or null output");
  return qsa_attn_launch(g, a, 1, partials, p0, p1, CR_OUT_RAW_F32, (cudaStream_t)stream);
}

extern "C" cr_status cr_qsa_merge_partials(const cr_geometry* g, const cr_qsa_args* a, int ranks, const float* partials,
                                           cr_out_format fmt, void* stream) {
  using namespace cr;
  if (cr_status s = qsa_validate(g, a, 1, CR_MAX_PREFILL_ROWS, "cr_qsa_merge_partials", 0)) return s;
  if (cr_status s = check_out(a, 1, fmt, "cr_qsa_merge_partials")) return s;
  CR_REQUIRE(partials && ranks >= 1 && ranks <= 32, "cr_qsa_merge_partials: need gathered partials of 1..32 ranks");
  return qsa_merge_launch(g, *a, ranks, partials, fmt, (cudaStream_t)stream);
}

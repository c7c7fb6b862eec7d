// Gated DeltaNet decode / speculative-verify step for sm_100a.
//
// A cluster of 1, 2 or 4 CTAs of 8 warps per (value head, span).  The delta rule never mixes value columns, so a CTA has its
// share of the columns of the head's 128 x 128 fp32 state and a warp 16 of them (8 in clusters); a lane holds 4 (2) columns x 16
// keys in registers (as pairs of keys, for the two-lane fp32 instructions), so a row of the pass costs a warp eight 128-bit
// reads of shared memory, eleven (nine) shuffles and no barrier, and the rows (replayed ones first) run back to back.
// Everything the pass reads is asked for at the start: raw rows with their halo and the pending rows into shared memory, the
// state into L2 and, behind the a / b dot products, into registers, the gate rows during the recurrence.  The CTAs of a cluster
// prepare the same rows; what they exchange is the readout, once, for the norm over the head's columns.
//
// Semantics follow GdnKernel (engine/layers/ops.h:252-401): replay of pending rows, per-row update with the
// readout from the updated state, state stored after row commit-1, rows >= commit recorded as
// (khat, v, decay, beta), gated RMSNorm readout, raw-row ring update.
//
// Bound: latency of a few dependent memory round trips; with many rows the update chain.  Reads of k and q from shared memory
// set the pace of every form with less state per lane: 8 sessions x (9 rows + 4 replayed), 32 heads, took 95 us with a quarter
// of the columns per CTA and two barriers a row, 52 us with 8 columns per warp and none, 32 us now.  One session x 1 row, 32
// heads, state in L2 / in HBM: 6.8 / 9.2 us in that first form, 8.6 / 9.1 on a CTA per head, which pulls 64 KB of state, 6.6 / 7.1
// as clusters of four.  4 sessions x 1 row: 9.8 / 12.9, now 8.8 / 10.1.  (Plain launches; chained ones take 0.5 to 0.8 less.)
//
// Prefill calls of up to 26 rows run here as well, 13 at most to a launch: their rows come in fp32 or bf16 with a and b as logits, all of
// them are committed, and nothing is replayed.
#include <cooperative_groups.h>
#include "gdn_prefill.cuh"

namespace cg = cooperative_groups;

namespace cr {

constexpr int kStepRows = CR_MAX_STEP_ROWS;
constexpr int kStepThreads = 256, kStepWarps = kStepThreads / 32;
constexpr int kReplayChunk = 16;                       // pending rows staged at a time
constexpr int kRawCols = 384;                          // channels of a head: 128 q, 128 k, 128 v

struct GdnStepParams {
  cr_gdn_args span[kMaxSpans];
  int Hv, Hk, hidden, pend_rows, fmt;
  int rows, replay;                                    // most of any span: the shared-memory layout
  const void* logits;                                  // rows of a prefill call: [R][2 Hv] a and b logits in the place of x and ab
  float* raw_y;                                        // and, where it is asked for, [R][Hv * 128] of un-gated readout
};
// What a pass reads: the rows of a step (fp32 projections, a and b from dot products with x), or those of a short prefill call
// (projections and logits in fp32 or bf16).
enum StepInput { kStepRowsIn, kPrefillF32, kPrefillBf16 };

// Floats of dynamic shared memory: raw rows with halo, q, k and v rows (the readout replaces v), staged pending rows.
__host__ __device__ constexpr int step_smem_floats(int rows, int replay) {
  const int rep = replay < kReplayChunk ? replay : kReplayChunk;
  return (rows + 3) * kRawCols + rows * kRawCols + rep * 258;
}

template <int BYTES>
__device__ __forceinline__ void step_cp(float* dst, const float* src, bool valid) {
  const int bytes = valid ? BYTES : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "n"(BYTES), "r"(bytes));
}

// A head is a cluster of CL CTAs (grid x: CL per head); CTA k has 128 / CL of its value columns, NC of them per lane.
template <int CL, int IN>
__global__ void __launch_bounds__(kStepThreads, 2) gdn_step_kernel(const __grid_constant__ GdnStepParams P) {
  constexpr int NC = CL == 1 ? 4 : 2, kWarpCols = 4 * NC, kOwners = 128 / CL / kWarpCols;   // columns of a lane, of a warp; warps that own columns
  extern __shared__ __align__(16) float step_sm[];
  __shared__ float ab_warp[kStepWarps][kStepRows][2];          // a / b dot products by warp
  __shared__ float dec[kStepRows], bet[kStepRows];
  const cr_gdn_args& a = P.span[blockIdx.y];
  const int h = blockIdx.x / CL, rank = blockIdx.x % CL, t = threadIdx.x, w = t >> 5, l = t & 31;
  const int kg = l & 7, col = rank * (128 / CL) + kWarpCols * w + NC * (l >> 3);   // keys 32 i + 4 kg + j of the columns col .. col + NC - 1
  const int own = NC == 4 ? (l & 1) * 2 + ((l >> 1) & 1) : l & 1;                  // the column (of the NC) whose sums end up in this lane
  const bool owner = kOwners == kStepWarps || w < kOwners;
  const int rep = P.Hv / P.Hk, kh = h / rep, KW = P.Hk * 128, VW = P.Hv * 128, C = 2 * KW + VW;
  const int R = a.R;
  float* raw = step_sm;                                        // [R + 3][384]: rows -3 .. R - 1
  float* qs = raw + (P.rows + 3) * kRawCols;                   // [R][128]
  float* ks = qs + P.rows * 128;
  float* vs = ks + P.rows * 128;                               // a column's y replaces its v once that has been read
  float* pk = vs + P.rows * 128;                               // staged pending rows: keys | values, then (decay, beta)
  float* pg = pk + min(P.replay, kReplayChunk) * 256;
  constexpr bool BF = IN == kPrefillBf16;
  pdl_release();
  touch_params(a);
  pdl_wait();

  // ---- everything the pass reads is asked for: state (L2), raw rows and pending rows (shared memory)
  float* st = a.state + (size_t)h * 16384;
#pragma unroll
  for (int i = 0; i < 2 / CL + (CL > 2); ++i)                  // 128 / CL columns of the 128 rows, 128 bytes at a time
    if (CL < 4 || t < 128) {
      const int line = t + 256 * i;
      asm volatile("prefetch.global.L2 [%0];\n" ::"l"(st + (size_t)(line / (4 / CL)) * 128 + rank * (128 / CL) + line % (4 / CL) * 32));
    }
  const float* qkv = reinterpret_cast<const float*>(a.qkv);
  {
    // a warp takes every eighth row, a lane the same channels of each: 96 pieces of 4 channels, or 384 single ones
    const bool vec = (((uintptr_t)qkv | (uintptr_t)a.hist) & 15) == 0;
    const int per = vec ? kRawCols / 4 : kRawCols;
    for (int rr = w; rr < R + 3; rr += kStepWarps) {
      const int p = a.pos0 + rr - 3;
      if (BF && rr >= 3) {
        for (int c = l; c < kRawCols; c += 32)
          raw[rr * kRawCols + c] = load_in<BF>(a.qkv, (long long)(rr - 3) * C + (c < 128 ? kh * 128 + c : (c < 256 ? KW + kh * 128 + c - 128 : 2 * KW + h * 128 + c - 256)));
        continue;
      }
      const float* row = rr >= 3 ? qkv + (size_t)(rr - 3) * C : a.hist + (size_t)(p & 15) * C;
      for (int i = l; i < per; i += 32) {
        const int c = vec ? 4 * i : i;
        const float* src = row + (c < 128 ? kh * 128 + c : (c < 256 ? KW + kh * 128 + c - 128 : 2 * KW + h * 128 + c - 256));
        if (vec) step_cp<16>(raw + rr * kRawCols + c, src, p >= 0);
        else step_cp<4>(raw + rr * kRawCols + c, src, p >= 0);
      }
    }
  }
  auto stage_pending = [&](int i0, int n) {
    for (int i = w; i < n; i += kStepWarps) {
      const float* pe = a.pend + ((size_t)h * P.pend_rows + i0 + i) * CR_PEND_FLOATS;
      for (int c = l; c < 258; c += 32) step_cp<4>(c < 256 ? pk + i * 256 + c : pg + 2 * i + c - 256, pe + c, true);
    }
  };
  if (a.replay > 0) stage_pending(0, min(a.replay, kReplayChunk));
  asm volatile("cp.async.commit_group;\n" ::: "memory");

  // ---- a / b dot products: all threads on one row, or four groups of 64 threads on every fourth row
  const int groups = R == 1 ? 1 : 4, lanes = kStepThreads / groups, grp = t / lanes;
  float la = 0.f, lb = 0.f;                                    // a prefill call brings them along: row t
  if (IN != kStepRowsIn) {
    if (t < R) { la = load_in<BF>(P.logits, (long long)t * 2 * P.Hv + h); lb = load_in<BF>(P.logits, (long long)t * 2 * P.Hv + P.Hv + h); }
  } else {
    constexpr int kMost = (kStepRows + 3) / 4;                 // rows of a group
    f2 pa[kMost], pb[kMost];
#pragma unroll
    for (int k = 0; k < kMost; ++k) pa[k] = pb[k] = 0ull;
    const __half* wa = reinterpret_cast<const __half*>(a.ab) + (size_t)h * P.hidden;
    const __half* wb = reinterpret_cast<const __half*>(a.ab) + (size_t)(P.Hv + h) * P.hidden;
#pragma unroll 2
    for (int u = t & (lanes - 1); u < P.hidden / 8; u += lanes) {
      const uint4 ua = *reinterpret_cast<const uint4*>(wa + u * 8), ub = *reinterpret_cast<const uint4*>(wb + u * 8);
      const __half2* ha = reinterpret_cast<const __half2*>(&ua);
      const __half2* hb = reinterpret_cast<const __half2*>(&ub);
      f2 fa[4], fb[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 x = __half22float2(ha[j]), y = __half22float2(hb[j]);
        fa[j] = pack2(x.x, x.y); fb[j] = pack2(y.x, y.y);
      }
#pragma unroll
      for (int k = 0; k < kMost; ++k) {
        const int r = grp + 4 * k;
        if (r >= R) break;
        f2 x[4];
        load_f2x2(a.x + (size_t)r * P.hidden + u * 8, x[0], x[1]);
        load_f2x2(a.x + (size_t)r * P.hidden + u * 8 + 4, x[2], x[3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) { pa[k] = fma2(fa[j], x[j], pa[k]); pb[k] = fma2(fb[j], x[j], pb[k]); }
      }
    }
#pragma unroll
    for (int k = 0; k < kMost; ++k) {
      const int r = grp + 4 * k;
      if (r >= R) break;
      const float2 xa = unpack2(pa[k]), xb = unpack2(pb[k]);
      const float sa = warp_sum(xa.x + xa.y), sb = warp_sum(xb.x + xb.y);
      if (l == 0) { ab_warp[w][r][0] = sa; ab_warp[w][r][1] = sb; }
    }
  }
  // The state, from L2 by now: its registers are not needed while the dot products hold theirs.
  f2 S[NC][8];                                                 // [column][pair of keys 32 (m / 2) + 4 kg + 2 (m % 2)]
  if (owner) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float* s2 = st + (size_t)(32 * (i >> 1) + 4 * kg + 2 * (i & 1)) * 128 + col;
      if constexpr (NC == 4) {
        const float4 x = *reinterpret_cast<const float4*>(s2), y = *reinterpret_cast<const float4*>(s2 + 128);
        S[0][i] = pack2(x.x, y.x); S[1][i] = pack2(x.y, y.y); S[2][i] = pack2(x.z, y.z); S[3][i] = pack2(x.w, y.w);
      } else {
        const float2 x = *reinterpret_cast<const float2*>(s2), y = *reinterpret_cast<const float2*>(s2 + 128);
        S[0][i] = pack2(x.x, y.x); S[1][i] = pack2(x.y, y.y);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();

  // The sums over the eight key groups of NC values per lane: every lane ends up with that of its own column.  A column's sum
  // has the same order for every NC, so a pass gives the same bits whatever else shares its launch.
  auto reduce = [&](const float (&x)[NC]) {
    const bool hi = l & 1;
    float s;
    if constexpr (NC == 4) {
      const bool odd = l & 2;
      float a0 = hi ? x[2] : x[0], a1 = hi ? x[3] : x[1];
      a0 += __shfl_xor_sync(0xffffffffu, hi ? x[0] : x[2], 1);
      a1 += __shfl_xor_sync(0xffffffffu, hi ? x[1] : x[3], 1);
      s = (odd ? a1 : a0) + __shfl_xor_sync(0xffffffffu, odd ? a0 : a1, 2);
    } else {
      s = (hi ? x[1] : x[0]) + __shfl_xor_sync(0xffffffffu, hi ? x[0] : x[1], 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
    }
    return s + __shfl_xor_sync(0xffffffffu, s, 4);
  };
  // One delta-rule update with the 128 key values kv and the head's value row v; the readout of the updated state goes over
  // v where qv is given.
  auto update = [&](const float* kv, const float* qv, float decay, float beta, float* v) {
    if (!owner) return;
    f2 k2[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) load_f2x2(kv + 32 * i + 4 * kg, k2[2 * i], k2[2 * i + 1]);
    auto columns = [&](float (&m)[NC]) {                        // this lane's share of k2 . S
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        f2 x = mul2(S[c][0], k2[0]), y = mul2(S[c][1], k2[1]);
#pragma unroll
        for (int i = 2; i < 8; i += 2) { x = fma2(S[c][i], k2[i], x); y = fma2(S[c][i + 1], k2[i + 1], y); }
        const float2 z = unpack2(add2(x, y));
        m[c] = z.x + z.y;
      }
    };
    float m[NC];
    columns(m);
    const float mine = beta * (v[col + own] - decay * reduce(m));
    float delta[NC];                                            // back to every lane
    if constexpr (NC == 4) {
      const float pair = __shfl_xor_sync(0xffffffffu, mine, 2);
      const float d0 = (l & 2) ? pair : mine, d1 = (l & 2) ? mine : pair;
      const float e0 = __shfl_xor_sync(0xffffffffu, d0, 1), e1 = __shfl_xor_sync(0xffffffffu, d1, 1);
      delta[0] = (l & 1) ? e0 : d0; delta[1] = (l & 1) ? e1 : d1; delta[2] = (l & 1) ? d0 : e0; delta[3] = (l & 1) ? d1 : e1;
    } else {
      const float other = __shfl_xor_sync(0xffffffffu, mine, 1);
      delta[0] = (l & 1) ? other : mine; delta[1] = (l & 1) ? mine : other;
    }
    const f2 g2 = pack2(decay, decay);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const f2 d2 = pack2(delta[c], delta[c]);
#pragma unroll
      for (int i = 0; i < 8; ++i) S[c][i] = fma2(k2[i], d2, mul2(g2, S[c][i]));
    }
    if (qv) {
#pragma unroll
      for (int i = 0; i < 4; ++i) load_f2x2(qv + 32 * i + 4 * kg, k2[2 * i], k2[2 * i + 1]);
      columns(m);
      const float y = reduce(m);
      if (kg < NC) v[col + own] = y;                            // the warp has read its v before the shuffles
    }
  };

  // ---- lazy commit: fold the accepted rows of the previous pass into the state (no readout)
  for (int i0 = 0; i0 < a.replay; i0 += kReplayChunk) {
    const int n = min(a.replay - i0, kReplayChunk);
    if (i0 > 0) {
      __syncthreads();                                         // the chunk before has been used
      stage_pending(i0, n);
      asm volatile("cp.async.commit_group;\n" ::: "memory");
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      __syncthreads();
    }
    for (int i = 0; i < n; ++i) update(pk + i * 256, nullptr, pg[2 * i], pg[2 * i + 1], pk + i * 256 + 128);
  }
  if (CL > 1 && a.replay > 0 && R > a.commit) cg::this_cluster().sync();   // every CTA has its pending rows before new ones are recorded

  // ---- conv + SiLU: a thread takes q or k channel t of all rows and a v channel of every other row
  {
    const float4 wqk = *reinterpret_cast<const float4*>(a.conv + (size_t)((t < 128 ? 0 : KW - 128) + kh * 128 + t) * 4);
    const float4 wv = *reinterpret_cast<const float4*>(a.conv + (size_t)(2 * KW + h * 128 + (t & 127)) * 4);
    auto conv = [&](const float4& c, float x0, float x1, float x2, float x3) {
      float s = c.x * x0;
      s = fmaf(c.y, x1, s);
      s = fmaf(c.z, x2, s);
      s = fmaf(c.w, x3, s);
      return siluf_(s);
    };
    float* dst = t < 128 ? qs + t : ks + t - 128;
    float x0 = raw[t], x1 = raw[kRawCols + t], x2 = raw[2 * kRawCols + t];
#pragma unroll 4
    for (int r = 0; r < R; ++r) {
      const float x3 = raw[(r + 3) * kRawCols + t];
      dst[r * 128] = conv(wqk, x0, x1, x2, x3);
      x0 = x1; x1 = x2; x2 = x3;
    }
    for (int r = t >> 7; r < R; r += 2) {
      const float* x = raw + r * kRawCols + 256 + (t & 127);
      vs[r * 128 + (t & 127)] = conv(wv, x[0], x[kRawCols], x[2 * kRawCols], x[3 * kRawCols]);
    }
  }
  __syncthreads();
  for (int i = w; i < 2 * R; i += kStepWarps) {                // a warp normalises a row of q or k
    float4* row = reinterpret_cast<float4*>((i < R ? qs + i * 128 : ks + (i - R) * 128) + 4 * l);
    const float4 x = *row;
    const float sc = rsqrtf(warp_sum(x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w) + kEps) * (i < R ? kInvSqrt128 : 1.f);
    *row = make_float4(x.x * sc, x.y * sc, x.z * sc, x.w * sc);
  }
  if (t < R) {
    float pa = la, pb = lb;
    if (IN == kStepRowsIn) {
      const int per = kStepWarps / groups, w0 = R == 1 ? 0 : (t & 3) * per;
      for (int k = w0; k < w0 + per; ++k) { pa += ab_warp[k][t][0]; pb += ab_warp[k][t][1]; }
    }
    const float sp = pa + a.dt_bias[h];
    const float softplus = sp > 20.f ? sp : log1pf(expf(sp));
    dec[t] = expf(-__expf(a.A_log[h]) * softplus);
    bet[t] = sigmoidf_(pb);
  }
  constexpr int kGateRows = (kStepRows + CL * kStepWarps - 1) / (CL * kStepWarps);
  float z[kGateRows][4];                                       // this warp's gate rows: in flight during the recurrence
#pragma unroll
  for (int k = 0; k < kGateRows; ++k) {
    const int r = rank + CL * (w + kStepWarps * k);
#pragma unroll
    for (int i = 0; i < 4; ++i) z[k][i] = r < R ? load_in<BF>(a.z, (long long)r * VW + h * 128 + 4 * l + i) : 0.f;
  }
  __syncthreads();

  // ---- raw-row ring (slots of this call never alias the three slots any CTA reads: R + 3 <= 16) and speculative rows:
  // (khat, v, decay, beta) for the next pass's replay, whose old rows every warp of this head has used
  for (int r = rank + CL * w; r < R; r += CL * kStepWarps) {
    float* hs = a.hist + (size_t)((a.pos0 + r) & 15) * C;
    const float* x = raw + (r + 3) * kRawCols;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = l + 32 * i;
      hs[2 * KW + h * 128 + c] = x[256 + c];
      if (h % rep == 0) { hs[kh * 128 + c] = x[c]; hs[KW + kh * 128 + c] = x[128 + c]; }
    }
    if (r >= a.commit) {
      float* pe = a.pend + ((size_t)h * P.pend_rows + (r - a.commit)) * CR_PEND_FLOATS;
#pragma unroll
      for (int i = 0; i < 4; ++i) { pe[l + 32 * i] = ks[r * 128 + l + 32 * i]; pe[128 + l + 32 * i] = vs[r * 128 + l + 32 * i]; }
      if (l < 2) pe[256 + l] = l == 0 ? dec[r] : bet[r];
    }
  }
  if (R > a.commit) __syncthreads();                           // the readout overwrites v

  // ---- the recurrence
  for (int r = 0; r < R; ++r) {
    update(ks + r * 128, qs + r * 128, dec[r], bet[r], vs + r * 128);
    if (owner && r == a.commit - 1) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float2 x[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) x[c] = unpack2(S[c][i]);
        float* s2 = st + (size_t)(32 * (i >> 1) + 4 * kg + 2 * (i & 1)) * 128 + col;
        if constexpr (NC == 4) {
          *reinterpret_cast<float4*>(s2) = make_float4(x[0].x, x[1].x, x[2].x, x[3].x);
          *reinterpret_cast<float4*>(s2 + 128) = make_float4(x[0].y, x[1].y, x[2].y, x[3].y);
        } else {
          *reinterpret_cast<float2*>(s2) = make_float2(x[0].x, x[1].x);
          *reinterpret_cast<float2*>(s2 + 128) = make_float2(x[0].y, x[1].y);
        }
      }
    }
  }
  if constexpr (CL == 1) __syncthreads();
  else cg::this_cluster().sync();                              // the readout of all columns is there

  // ---- gated RMSNorm over the head's 128 columns, a warp per row (the rows dealt over the cluster), lane l the columns 4 l .. 4 l + 3
  const float* yv_s = CL == 1 ? vs : cg::this_cluster().map_shared_rank(vs, l * CL / 32);
#pragma unroll
  for (int k = 0; k < kGateRows; ++k) {
    const int r = rank + CL * (w + kStepWarps * k);
    if (r >= R) break;
    const float4 y = *reinterpret_cast<const float4*>(yv_s + r * 128 + 4 * l);
    const float rs = rsqrtf(warp_sum(y.x * y.x + y.y * y.y + y.z * y.z + y.w * y.w) * (1.f / 128.f) + kEps);
    const float yv[4] = {y.x, y.y, y.z, y.w};
    float o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = yv[i] * rs * a.gamma[4 * l + i] * sigmoidf_(z[k][i]);
    const size_t at = (size_t)r * VW + h * 128 + 4 * l;
    if (IN != kStepRowsIn && P.raw_y) *reinterpret_cast<float4*>(P.raw_y + at) = y;
    if (P.fmt == CR_OUT_RAW_F32) {
      float* dst = reinterpret_cast<float*>(a.out) + at;
      if (((uintptr_t)dst & 15) == 0) *reinterpret_cast<float4*>(dst) = make_float4(o[0], o[1], o[2], o[3]);
      else { dst[0] = o[0]; dst[1] = o[1]; dst[2] = o[2]; dst[3] = o[3]; }
    } else if (P.fmt == CR_OUT_RAW_BF16) {
      __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(a.out) + at;
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        const __nv_bfloat162 b = __floats2bfloat162_rn(o[i], o[i + 1]);
        if (((uintptr_t)dst & 3) == 0) *reinterpret_cast<__nv_bfloat162*>(dst + i) = b;
        else { dst[i] = b.x; dst[i + 1] = b.y; }
      }
    } else {
      float su[4];
      load_half4(a.suh_out + h * 128 + 4 * l, su);
#pragma unroll
      for (int i = 0; i < 4; ++i) o[i] = round_h(round_h(o[i]) * su[i]);
      wht128(o);
      store_half4(reinterpret_cast<uint16_t*>(a.out) + out_index(r, h * 128 + 4 * l, VW, a.pack_rows, a.pack_off), o, kHadNorm);
    }
  }
  if constexpr (CL > 1) cg::this_cluster().sync();             // the rows stay until every CTA has read them
}

// With more than half of an SM's shared memory a CTA has an SM of its own.  Calls that fit the SMs once ask for that: let in while
// the kernel ahead still holds most SMs, the CTAs would pair up on the free ones and stay there, and a pair takes half as long
// again (steps of 3 sessions x 1 row, 32 heads, one behind the other: 12.7 us paired, 9.0 us).
constexpr size_t kAloneSmem = 116 * 1024;
static_assert(step_smem_floats(kStepRows, kReplayChunk) * sizeof(float) <= kAloneSmem, "the longest pass fits");

template <int CL>
static cudaLaunchConfig_t step_config(dim3 grid, size_t smem, cudaStream_t stream, cudaLaunchAttribute (&attr)[2]) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = dim3(kStepThreads); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cfg.attrs = attr;
  if (CL > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = CL; attr[cfg.numAttrs].val.clusterDim.y = 1; attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  return cfg;
}
// Heads whose clusters of CL CTAs, an SM to each, the device holds at once (looked up once per device).
template <int CL, int IN>
static cr_status step_heads(int& heads) {
  static PerDeviceOnce looked_up;
  static int table[64];
  int dev = 0;
  CR_CUDA(cudaGetDevice(&dev));
  if (cr_status st = once_per_device(looked_up, [dev] {
        CR_CUDA(cudaFuncSetAttribute(gdn_step_kernel<CL, IN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAloneSmem));
        cudaLaunchAttribute attr[2];
        cudaLaunchConfig_t cfg = step_config<CL>(dim3(CL), kAloneSmem, nullptr, attr);
        if (CL > 1) CR_CUDA(cudaOccupancyMaxActiveClusters(&table[dev & 63], gdn_step_kernel<CL, IN>, &cfg));
        else table[dev & 63] = sm_count();
        return CR_OK;
      })) return st;
  heads = table[dev & 63];
  return CR_OK;
}
template <int CL, int IN>
static cr_status step_launch(const GdnStepParams& P, int n, bool alone, cudaStream_t stream) {
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = step_config<CL>(dim3(P.Hv * CL, n), alone ? kAloneSmem : step_smem_floats(P.rows, P.replay) * sizeof(float), stream, attr);
  if (pdl_enabled()) { attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1; }
  CR_CUDA(cudaLaunchKernelEx(&cfg, gdn_step_kernel<CL, IN>, P));
  CR_LAUNCH_CHECK("gdn_step_kernel");
  return CR_OK;
}

// Few heads leave SMs idle: a head is spread over as many CTAs as there are SMs for, all clusters at once.  States in HBM, 1 / 9
// rows: 32 heads 9.1 / 21.2 us on one CTA each, 8.0 / 18.3 on two, 7.1 / 17.3 on four; 64 heads 9.3 / 21.7, 8.4 / 18.9, 8.6 / 19.8;
// 96 heads 9.7 / 22.1, 10.8 / 22.5: once two CTAs share an SM the work that a head's CTAs repeat (rows, dot products) costs more.
template <int IN>
static cr_status step_dispatch(const GdnStepParams& P, int n, cudaStream_t stream) {
  int fit4, fit2, fit1;
  if (cr_status st = step_heads<4, IN>(fit4)) return st;
  if (cr_status st = step_heads<2, IN>(fit2)) return st;
  if (cr_status st = step_heads<1, IN>(fit1)) return st;
  const int heads = n * P.Hv;
  const auto launch = heads <= fit4 ? step_launch<4, IN> : (heads <= fit2 ? step_launch<2, IN> : step_launch<1, IN>);
  return launch(P, n, heads <= fit1, stream);
}

// The rows of a prefill call of at most CR_MAX_STEP_ROWS rows through the recurrence: what bounds a call of one chunk is the chain of
// its phases, whatever its rows.
cr_status gdn_few_rows(const cr_geometry* g, const cr_gdn_args& a, const void* logits, float* raw_y, bool bf16_in, cr_out_format fmt, cudaStream_t stream) {
  GdnStepParams P;
  P.span[0] = a;
  P.Hv = g->gdn_vheads; P.Hk = g->gdn_kheads; P.hidden = g->hidden; P.pend_rows = 1; P.fmt = (int)fmt;
  P.rows = a.R; P.replay = 0;
  P.logits = logits; P.raw_y = raw_y;
  return bf16_in ? step_dispatch<kPrefillBf16>(P, 1, stream) : step_dispatch<kPrefillF32>(P, 1, stream);
}

}  // namespace cr

extern "C" cr_status cr_gdn_step(const cr_geometry* g, const cr_gdn_args* spans, int n_spans, int pend_rows,
                                 cr_out_format fmt, void* stream) {
  using namespace cr;
  if (cr_status s = check_geometry(g)) return s;
  CR_REQUIRE(spans && n_spans >= 1, "cr_gdn_step: no spans");
  use_stream((cudaStream_t)stream);
  CR_REQUIRE(pend_rows >= 1 && pend_rows <= 64, "cr_gdn_step: pend_rows %d out of range", pend_rows);
  CR_REQUIRE(fmt == CR_OUT_RAW_F32 || fmt == CR_OUT_RAW_BF16 || fmt == CR_OUT_EXL3_WHT, "cr_gdn_step: bad output format");
  for (int s = 0; s < n_spans; ++s) {
    const cr_gdn_args& a = spans[s];
    CR_REQUIRE(a.R >= 1 && a.R <= CR_MAX_STEP_ROWS, "cr_gdn_step: span %d has R=%d, need 1..%d", s, a.R, CR_MAX_STEP_ROWS);
    CR_REQUIRE(a.pos0 >= 0, "cr_gdn_step: span %d has negative pos0", s);
    CR_REQUIRE(a.commit >= 1 && a.commit <= a.R, "cr_gdn_step: span %d commit=%d must be in 1..R (a verify pass keeps at least one row)", s, a.commit);
    CR_REQUIRE(a.replay >= 0 && a.replay <= pend_rows, "cr_gdn_step: span %d replay=%d exceeds the pending rows", s, a.replay);
    CR_REQUIRE(a.R - a.commit <= pend_rows, "cr_gdn_step: span %d records %d pending rows, stride is %d", s, a.R - a.commit, pend_rows);
    CR_REQUIRE(a.qkv && a.z && a.x && a.ab && a.conv && a.A_log && a.dt_bias && a.gamma && a.hist && a.state && a.out,
               "cr_gdn_step: span %d has a null buffer", s);
    CR_REQUIRE(a.pend || (a.replay == 0 && a.commit == a.R), "cr_gdn_step: span %d needs a pending-row buffer", s);
    CR_REQUIRE(fmt != CR_OUT_EXL3_WHT || a.suh_out, "cr_gdn_step: span %d needs suh_out for the EXL3 output", s);
    CR_REQUIRE(fmt == CR_OUT_EXL3_WHT || a.pack_rows == 0, "cr_gdn_step: packed layout only with the EXL3 output");
  }
  for (int s0 = 0; s0 < n_spans; s0 += kMaxSpans) {
    GdnStepParams P;
    const int n = n_spans - s0 < kMaxSpans ? n_spans - s0 : kMaxSpans;
    for (int s = 0; s < n; ++s) P.span[s] = spans[s0 + s];
    P.Hv = g->gdn_vheads; P.Hk = g->gdn_kheads; P.hidden = g->hidden; P.pend_rows = pend_rows; P.fmt = (int)fmt;
    P.rows = P.replay = 0;
    P.logits = nullptr; P.raw_y = nullptr;
    for (int s = 0; s < n; ++s) {
      P.rows = P.rows > P.span[s].R ? P.rows : P.span[s].R;
      P.replay = P.replay > P.span[s].replay ? P.replay : P.span[s].replay;
    }
    if (cr_status st = step_dispatch<kStepRowsIn>(P, n, (cudaStream_t)stream)) return st;
  }
  return CR_OK;
}

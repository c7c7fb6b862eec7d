// gdn_chunk_local_kernel: everything of the chunk-64 WY scan that does not depend on the carried state, fully
// parallel over (chunk, key head).  Per CTA:
//   1. raw projection rows of the key head's q and k channels are staged in shared memory with cp.async (3 halo rows
//      from the previous rows, the ring, or zero; with bf16 inputs the next tile is always in flight while the
//      current one is used), then conv(4) + SiLU + L2 norm -> qhat, khat (tf32); the gates (log-decay prefix G, beta
//      and their exponential tables) of the value heads are computed while the first tiles arrive;
//   2. Gram matrices K K^T and Q K^T on tensor cores, kept in accumulator registers for all value heads;
//   3. per value head: K'^T = (e^{G_end - G} K)^T and e^G Q tiles, L = tril(beta K K^T e^{dG}, -1), QKd = tril(Q K^T e^{dG}), and
//      T = (I + L)^-1 by an exact fp32 blocked inverse (16 x 16 diagonal blocks by substitution, off-diagonal blocks
//      in block-row order), then W = T (beta e^G K) and Ut = T (beta V) on tensor cores with tf32 operands; the
//      v columns run conv + SiLU from the staged raw rows.
// Outputs go straight into the layouts the scan consumes (K-major tiles for the tcgen05 scan).
// Two CTAs of 16 warps fit per SM (113 KB of shared memory, 64 registers x 512 threads each).  With 8 warps each a phase
// lasted about as long alone on an SM as beside another CTA: latency of shuffles, shared-memory loads and barriers, not
// issue slots, set the pace.  With 16 warps, pairs of fp32 in one instruction, the norms taken from registers and products
// of the inverse reading both factors 16 bytes at a time the kernel issues 60 % of the time.  7,104 rows, 16 / 32 heads:
// 256 -> 232 us alone; 333 rows 36 -> 26 us; 64 rows 32 -> 16 us; 1,999 fp32 rows, 16 / 48 heads: 131 -> 120 us.
//
// The scan reads a chunk as soon as it is written: units are walked in chunk order and mark what they finish, and in a call of one
// part the scan's CTAs run beside this kernel, on SMs that it leaves to them.  The call then takes what the longer of the two
// takes, not their sum: 1,999 rows, 16 / 32 heads, 193 -> 156 us, 16 / 48 heads from fp32 rows 247 -> 225 us, 7,104 rows 570 ->
// 410 us.  The scan waits for this kernel and never the other way, and is let in when every CTA here is resident.
#include <algorithm>
#include "gdn_chunk.cuh"

namespace cr {

// The two halves of a CTA work on units of their own, each with its own barrier.
// (Read anew in every unit: addresses that the compiler keeps over the loop of units cost more registers than there are.)
__device__ __forceinline__ int local_tid() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t & 511;
}
__device__ __forceinline__ void local_sync() { asm volatile("bar.sync %0, 512;\n" ::"r"(1 + (int)(threadIdx.x >> 9)) : "memory"); }

constexpr int kCleared = 3;                                // barrier: the marks of the CTA are cleared
constexpr int kRawRows = 67;                               // 64 rows + 3 halo rows
constexpr int kStageBytes = kRawRows * 128 * 2;            // one 128-channel bf16 tile (or 64 fp32 channels)
constexpr int kLocalThreads = 512;
constexpr size_t kLocalSmem = (size_t)(64 * kLdK + 64 * kLdX + 64 * kLdM + 15 * 64 + 8 * 256) * sizeof(float) + kStageBytes + 256;

// Starts the copy of rows row0-3 .. row0+63 of channels [ch0, ch0+CH) into dst[67][CH] (element type of the input)
// as one cp.async group; rows past the end of the call are zero-filled.  Rows before the call come from the input
// itself (halo_in: a later part of one call), or, with plain stores, from the ring or zero.
template <bool BF16, int CH>
__device__ __forceinline__ void stage_issue(const GdnPrefillParams& P, int C, int row0, int ch0, void* dst) {
  constexpr int EPV = BF16 ? 8 : 4;                        // elements per 16-byte piece
  constexpr int PPR = CH / EPV;                            // pieces per row
  constexpr int RPP = kLocalThreads / PPR;                 // rows per pass
  const cr_gdn_args& a = P.a;
  const int pc = local_tid() % PPR, rr0 = local_tid() / PPR;
  uint4* d = reinterpret_cast<uint4*>(dst) + local_tid();
  const char* src = reinterpret_cast<const char*>(a.qkv) + ((long long)(row0 - 3 + rr0) * C + ch0 + pc * EPV) * (BF16 ? 2 : 4);
  const long long step = (long long)RPP * C * (BF16 ? 2 : 4);
#pragma unroll
  for (int k = 0; k * RPP < kRawRows; ++k, src += step) {
    const int rr = rr0 + k * RPP, r = row0 - 3 + rr;
    if ((k + 1) * RPP > kRawRows && rr >= kRawRows) break;
    if (r >= 0 || P.halo_in) {
      cp_async16(d + k * kLocalThreads, r < a.R ? src : reinterpret_cast<const char*>(a.qkv), r < a.R);
    } else {
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (a.pos0 + r >= 0) {
        const float* hs = a.hist + (size_t)((a.pos0 + r) & 15) * C + ch0 + pc * EPV;
        if constexpr (BF16) {
          __nv_bfloat162 b[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) b[i] = __floats2bfloat162_rn(hs[2 * i], hs[2 * i + 1]);
          v = *reinterpret_cast<const uint4*>(b);
        } else {
          v = make_uint4(__float_as_uint(hs[0]), __float_as_uint(hs[1]), __float_as_uint(hs[2]), __float_as_uint(hs[3]));
        }
      }
      d[k * kLocalThreads] = v;
    }
  }
  cp_async_commit();
}
template <bool BF16>
__device__ __forceinline__ f2 staged_pair(const void* buf, int CH, int rr, int ch) {
  if constexpr (BF16) {
    const unsigned v = *reinterpret_cast<const unsigned*>(reinterpret_cast<const __nv_bfloat16*>(buf) + rr * CH + ch);
    return pack2(__uint_as_float(v << 16), __uint_as_float(v & 0xFFFF0000u));
  } else {
    return *reinterpret_cast<const f2*>(reinterpret_cast<const float*>(buf) + rr * CH + ch);
  }
}

// conv(4) + SiLU of two channels (conv row ch, staged column col) over N rows from the staged rows of a tile.
template <bool BF16, int N>
__device__ __forceinline__ void conv_rows(const float* conv, int ch, const void* src, int CH, int row, int col, f2 (&out)[N]) {
  const float4 w0 = *reinterpret_cast<const float4*>(conv + (size_t)ch * 4), w1 = *reinterpret_cast<const float4*>(conv + (size_t)(ch + 1) * 4);
  const f2 t0 = pack2(w0.x, w1.x), t1 = pack2(w0.y, w1.y), t2 = pack2(w0.z, w1.z), t3 = pack2(w0.w, w1.w);
  f2 x0 = staged_pair<BF16>(src, CH, row, col), x1 = staged_pair<BF16>(src, CH, row + 1, col), x2 = staged_pair<BF16>(src, CH, row + 2, col);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const f2 x3 = staged_pair<BF16>(src, CH, row + 3 + i, col);       // staged row index = chunk row + 3
    const f2 c = fma2(t3, x3, fma2(t2, x2, fma2(t1, x1, mul2(t0, x0))));
    const float2 e = unpack2(mul2(c, pack2(-kLog2e, -kLog2e)));
    const float2 d = unpack2(add2(pack2(ex2_ftz(e.x), ex2_ftz(e.y)), pack2(1.f, 1.f)));
    out[i] = mul2(c, pack2(rcp_ftz(d.x), rcp_ftz(d.y)));
    x0 = x1; x1 = x2; x2 = x3;
  }
}
// Sums of eight values over the warp; lane l returns the sum of value l >> 2.
__device__ __forceinline__ float warp_sum8(float (&s)[8]) {
  const int l = threadIdx.x & 31;
#pragma unroll
  for (int k = 4; k >= 1; k >>= 1) {      // a lane keeps the half of the values that its bit of l >> 2 names
    const bool up = (l >> 2) & k;
#pragma unroll
    for (int i = 0; i < k; ++i) {
      const float keep = up ? s[i + k] : s[i], give = up ? s[i] : s[i + k];
      s[i] = keep + __shfl_xor_sync(0xffffffffu, give, 4 * k);
    }
  }
  float v = s[0];
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// T = (I + L)^-1 for the 64x64 unit lower-triangular I + L held in LT, in place, exact fp32, rounded to tf32 at the very
// end.  The diagonal 16 x 16 blocks come first (invert_diagonal: one thread per column by forward substitution, the two
// warps that do it need no barrier).  Then blocks (1,0) and (3,2), then the 32 x 32 block below the diagonal, each as
// T_ab = -T_aa (L_ab T_bb): a product per phase, all 512 threads busy.  What a product reads down a column is kept
// transposed as well, so that both factors come four to a load.
//
// Transposed 16 x 16 blocks: row j (a column of T), 16-byte unit u at u ^ (j / 2), free of bank conflicts for 16 rows.
__device__ __forceinline__ float* tr16(float* block, int j, int u) { return block + j * 16 + ((u ^ (j >> 1)) & 3) * 4; }
__device__ __forceinline__ void invert_diagonal(float* LT, float* Tt) {   // t < 64; Tt: T_00, T_11, T_22 and then T_10, transposed
  const int b = local_tid() >> 4, j = local_tid() & 15;
  float* B = LT + 16 * b * kLdM + 16 * b;
  float D[16];
#pragma unroll
  for (int r = 0; r < 16; ++r) {
    float acc = (r == j) ? 1.f : 0.f;
#pragma unroll
    for (int m = 0; m < r; ++m) acc = fmaf(-B[r * kLdM + m], D[m], acc);
    D[r] = acc;
  }
  __syncwarp();                          // both blocks of the warp have been read
#pragma unroll
  for (int r = 0; r < 16; ++r) B[r * kLdM + j] = D[r];
  if (b < 3)
#pragma unroll
    for (int u = 0; u < 4; ++u) *reinterpret_cast<float4*>(tr16(Tt + b * 256, j, u)) = make_float4(D[4 * u], D[4 * u + 1], D[4 * u + 2], D[4 * u + 3]);
}
// acc += sum over m < 16 of a[m] times row j of a transposed block, even and odd m apart
__device__ __forceinline__ f2 dot16(f2 acc, const float* a, float* block, int j) {
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    f2 a0, a1, b0, b1;
    load_f2x2(a + 4 * u, a0, a1);
    load_f2x2(tr16(block, j, u), b0, b1);
    acc = fma2(a1, b1, fma2(a0, b0, acc));
  }
  return acc;
}
__device__ __forceinline__ float sum2(f2 v) { const float2 x = unpack2(v); return x.x + x.y; }
__device__ __forceinline__ void round_quadrant(float* Q) {   // 32 x 32 at Q, two elements per thread
  float2* p = reinterpret_cast<float2*>(Q + (local_tid() >> 4) * kLdM + 2 * (local_tid() & 15));
  const float2 v = *p;
  *p = make_float2(tf32_operand(v.x), tf32_operand(v.y));
}
__device__ __forceinline__ void invert_unit_lower_64(float* LT, float* Tt, float* Ms) {   // after a barrier behind invert_diagonal
  const int t = local_tid(), half = t >> 8, i = (t >> 4) & 15, j = t & 15;
  auto put = [&](float* block, float v) { tr16(block, j, i >> 2)[i & 3] = v; };   // element (i, j)
  {
    const float* row = LT + (32 * half + 16 + i) * kLdM + 32 * half;
    put(Ms + half * 256, sum2(dot16(0ull, row, Tt + half * 512, j)));
    local_sync();
    const float v = -sum2(dot16(0ull, row + 16, Ms + half * 256, j));
    LT[(32 * half + 16 + i) * kLdM + 32 * half + j] = v;
    if (half == 0) put(Tt + 768, v);
    local_sync();
  }
  {   // a thread has rows 32 + i and 48 + i of one column; columns 16-31 meet a zero block of T in the first product
    const float *hi = LT + (32 + i) * kLdM, *lo = LT + (48 + i) * kLdM;
    f2 m0 = 0ull, m1 = 0ull;
    if (half == 0) { m0 = dot16(m0, hi, Tt, j); m1 = dot16(m1, lo, Tt, j); }
    float* below = Tt + (half == 0 ? 768 : 256);
    put(Ms + half * 512, sum2(dot16(m0, hi + 16, below, j)));
    put(Ms + half * 512 + 256, sum2(dot16(m1, lo + 16, below, j)));
    local_sync();
    const float t0 = -sum2(dot16(0ull, hi + 32, Ms + half * 512, j));
    const float t1 = -sum2(dot16(dot16(0ull, lo + 32, Ms + half * 512, j), lo + 48, Ms + half * 512 + 256, j));
    LT[(32 + i) * kLdM + 16 * half + j] = tf32_operand(t0);
    LT[(48 + i) * kLdM + 16 * half + j] = tf32_operand(t1);
    round_quadrant(LT);
    local_sync();
    round_quadrant(LT + 32 * kLdM + 32);
    local_sync();
  }
}

// Operands for the tcgen05 scan are written as K-major tiles float[K/4][rows][4] (plus Qt = e^G Q and K'^T).
// Chunk c, key head kh, value heads [v_first, v_last) of it.
template <bool BF16>
__device__ __forceinline__ void local_unit(const GdnPrefillParams& P, const ChunkWs& ws, float* sm, int c, int kh, int v_first, int v_last) {
  float* Ks = sm;                       // [64][132] khat (tf32)
  float* Qs = Ks + 64 * kLdK;           // [64][132] qhat (tf32), later [64][136] X = beta e^G K / beta V
  char* RB = reinterpret_cast<char*>(Qs + 64 * kLdX);      // raw staging tile
  float* LT = reinterpret_cast<float*>(RB + kStageBytes);  // [64][68] L, then T
  float* Gs = LT + 64 * kLdM;           // [3][64] cumulative log decay per value head
  float* bs = Gs + 3 * 64;              // [3][64] beta
  float* es = bs + 3 * 64;              // [3][64] beta * exp(G)
  float* egs = es + 3 * 64;             // [3][64] exp(G)
  float* scs = egs + 3 * 64;            // [3][64] exp(G_end - G)
  float* Ms = scs + 3 * 64;             // [4][16][16] scratch of the blocked inverse; first the partial sums of the L2 norms
  float* Tt = Ms + 4 * 256;             // [4][16][16] blocks of T, transposed
  const cr_gdn_args& a = P.a;
  const int t = local_tid(), w = t >> 5, l = t & 31, g = l >> 2, tq = l & 3;
  const int R = a.R, r0 = c * kChunk, valid = min(kChunk, R - r0);
  const int rep = P.Hv / P.Hk, KW = P.Hk * 128, VW = P.Hv * 128, C = 2 * KW + VW;
  constexpr int VCH = BF16 ? 128 : 64;  // channels of v per staging round

  // ---- 1. q and k of the key head, raw rows of both in flight at once: bf16 rows of q in the staging tile and of k in
  // the (still unused) L tile; fp32 rows of q as two 64-channel halves in those two and of k in the place of qhat.
  char* RB2 = reinterpret_cast<char*>(LT);
  if constexpr (BF16) {
    stage_issue<true, 128>(P, C, r0, kh * 128, RB);
    stage_issue<true, 128>(P, C, r0, KW + kh * 128, RB2);
  } else {
    stage_issue<false, 64>(P, C, r0, kh * 128, RB);
    stage_issue<false, 64>(P, C, r0, kh * 128 + 64, RB2);
    stage_issue<false, 128>(P, C, r0, KW + kh * 128, Qs);
  }
  // Gates while the first tiles are in flight: g = -exp(A_log) softplus(a + dt_bias), beta = sigmoid(b), prefix sum of
  // g inside the chunk; one warp per value head.  The tables are read after later barriers.
  if (w >= v_first && w < v_last) {
    const int h = kh * rep + w;
    const float A = -expf(a.A_log[h]), dtb = a.dt_bias[h];
    float gv[2], bv[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = 2 * l + k;
      gv[k] = 0.f; bv[k] = 0.f;
      if (i < valid) {
        const float sp = load_in<BF16>(P.ab_logits, (long long)(r0 + i) * 2 * P.Hv + h) + dtb;
        gv[k] = A * (sp > 20.f ? sp : log1pf(expf(sp)));
        bv[k] = sigmoidf_(load_in<BF16>(P.ab_logits, (long long)(r0 + i) * 2 * P.Hv + P.Hv + h));
      }
    }
    float s = gv[0] + gv[1];
#pragma unroll
    for (int step = 1; step < 32; step <<= 1) {
      const float v = __shfl_up_sync(0xffffffffu, s, step);
      if (l >= step) s += v;
    }
    const float G1 = s, G0 = s - gv[1];
    float* Gw = Gs + w * 64; float* bw = bs + w * 64; float* ew = es + w * 64;
    Gw[2 * l] = G0; Gw[2 * l + 1] = G1; bw[2 * l] = bv[0]; bw[2 * l + 1] = bv[1];
    const float e0 = __expf(G0), e1 = __expf(G1), Gend = __shfl_sync(0xffffffffu, G1, 31);
    ew[2 * l] = bv[0] * e0; ew[2 * l + 1] = bv[1] * e1;
    egs[w * 64 + 2 * l] = e0; egs[w * 64 + 2 * l + 1] = e1;
    scs[w * 64 + 2 * l] = __expf(Gend - G0); scs[w * 64 + 2 * l + 1] = __expf(Gend - G1);
    float* Gg = ws.G + ((size_t)h * ws.chunks + c) * 64;
    Gg[2 * l] = G0; Gg[2 * l + 1] = G1;
  }
  // A thread has two channels of eight rows, of q and of k: conv, SiLU and its share of the row sums stay in registers
  // until the two warps that share a row have exchanged their sums.
  const int pair = t & 63, rb = (t >> 6) * 8, ch2 = 2 * pair;
  f2 val[2][8];
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    if (part == 0) cp_async_wait_but_one(); else cp_async_wait_all();   // k is the last group
    local_sync();
    if constexpr (BF16) conv_rows<true>(a.conv, (part ? KW : 0) + kh * 128 + ch2, part ? RB2 : RB, 128, rb, ch2, val[part]);
    else if (part) conv_rows<false>(a.conv, KW + kh * 128 + ch2, Qs, 128, rb, ch2, val[1]);
    else conv_rows<false>(a.conv, kh * 128 + ch2, pair < 32 ? RB : RB2, 64, rb, ch2 & 63, val[0]);
    float s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = sum2(mul2(val[part][i], val[part][i]));
    const float sum = warp_sum8(s);     // of row rb + (l >> 2)
    if ((l & 3) == 0) Ms[part * 128 + (rb + (l >> 2)) * 2 + (w & 1)] = sum;
  }
  local_sync();
  // The raw rows have been read: v of the first value head may come in.
  stage_issue<BF16, VCH>(P, C, r0, 2 * KW + (kh * rep + v_first) * 128, RB);
  // L2 norms, scale, round to tf32; rows past the end are zero.  Lane 8 part + i has the factor of row rb + i.
  const float2 sums = *reinterpret_cast<const float2*>(Ms + (l >> 3 & 1) * 128 + (rb + (l & 7)) * 2);
  const float norm = rb + (l & 7) < valid ? rsqrt_ftz(sums.x + sums.y + kEps) * (l & 8 ? 1.f : kInvSqrt128) : 0.f;
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    float* dst = part ? Ks : Qs;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float sc = __shfl_sync(0xffffffffu, norm, 8 * part + i);
      const float2 o = unpack2(mul2(val[part][i], pack2(sc, sc)));
      *reinterpret_cast<float2*>(dst + (rb + i) * kLdK + ch2) = make_float2(tf32r(o.x), tf32r(o.y));
    }
  }
  local_sync();
  // per value head: K'^T = (e^{G_end - G} K)^T, K-major over tokens (unit (token / 4, key) holds 4 tokens of one
  // key; the decay towards the chunk end is folded into K so that the scan multiplies U itself), and
  // Qt = e^G Q, K-major over keys
  for (int vi = v_first; vi < v_last; ++vi) {
    float* kt = ws.Kt + ((size_t)(kh * rep + vi) * ws.chunks + c) * 8192;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int key = t & 127, tc = (t >> 7) + 4 * k;
      const float4 sc = *reinterpret_cast<const float4*>(scs + vi * 64 + 4 * tc);
      const float* K = Ks + 4 * tc * kLdK + key;
      *reinterpret_cast<float4*>(kt + (size_t)(tc * 128 + key) * 4) =
          make_float4(tf32_operand(sc.x * K[0]), tf32_operand(sc.y * K[kLdK]), tf32_operand(sc.z * K[2 * kLdK]), tf32_operand(sc.w * K[3 * kLdK]));
    }
    float* qt = ws.WQ + ((size_t)(kh * rep + vi) * ws.chunks + c) * 16384;
    const int row = t & 63;
    const float e = egs[vi * 64 + row];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int kc = (t >> 6) + 8 * k;
      const float4 q = *reinterpret_cast<const float4*>(Qs + row * kLdK + kc * 4);
      *reinterpret_cast<float4*>(qt + (size_t)(kc * 128 + 64 + row) * 4) = make_float4(tf32_operand(e * q.x), tf32_operand(e * q.y), tf32_operand(e * q.z), tf32_operand(e * q.w));
    }
  }
  // ---- 2. Gram matrices stay in registers: K K^T in warps 0-3 and 8-11, Q K^T in the others, 16 rows and 32 columns each;
  // the row blocks are dealt so that every scheduler gets one of each.
  const int mt = (w + (w >> 2)) & 3, n_first = (w >> 3) * 4;
  const bool is_kk = (w & 4) == 0;
  float gram[4][4];
#pragma unroll
  for (int n = 0; n < 4; ++n) gram[n][0] = gram[n][1] = gram[n][2] = gram[n][3] = 0.f;
  const int n_used = 2 * mt + 2 - n_first;   // column tiles at or below the diagonal of row block mt; the rest is masked
  if (n_used > 0) warp_gemm_nk_ldm<4, 16>(gram, (is_kk ? Ks : Qs) + mt * 16 * kLdK, kLdK, Ks + n_first * 8 * kLdK, kLdK, n_used);

  // ---- 3. per value head
  for (int vi = v_first; vi < v_last; ++vi) {
    const int h = kh * rep + vi;
    const size_t unit = (size_t)h * ws.chunks + c;
    const float* Gv = Gs + vi * 64; const float* bv = bs + vi * 64; const float* ev = es + vi * 64;
    local_sync();                    // previous head done with LT and X; qhat no longer needed
    {   // L and QKd straight from the Gram fragments
      float* qkd = ws.QKp + unit * 4096;
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int hrow = 0; hrow < 2; ++hrow) {
          const int row = mt * 16 + g + 8 * hrow, col = (n_first + n) * 8 + 2 * tq;
          if (n >= n_used) {            // above the diagonal: nothing reads L there, QKd is zero
            if (!is_kk) *reinterpret_cast<float2*>(qkd + ((col >> 2) * 64 + row) * 4 + (col & 3)) = make_float2(0.f, 0.f);
            continue;
          }
          const float Gr = Gv[row];
          const float p0 = ex2_ftz(fminf(Gr - Gv[col], 0.f) * kLog2e), p1 = ex2_ftz(fminf(Gr - Gv[col + 1], 0.f) * kLog2e);
          const float v0 = gram[n][2 * hrow], v1 = gram[n][2 * hrow + 1];
          if (is_kk) {
            const float b = bv[row];
            *reinterpret_cast<float2*>(LT + row * kLdM + col) = make_float2(col < row ? b * v0 * p0 : 0.f, col + 1 < row ? b * v1 * p1 : 0.f);
          } else {
            const int at = ((col >> 2) * 64 + row) * 4 + (col & 3);
            *reinterpret_cast<float2*>(qkd + at) = make_float2(col <= row ? tf32_operand(v0 * p0) : 0.f, col + 1 <= row ? tf32_operand(v1 * p1) : 0.f);
          }
        }
    }
    local_sync();
    if (w < 2) invert_diagonal(LT, Tt);
    else {
      for (int row = w - 2; row < 64; row += 14) {   // X = beta e^G K
        const int c4 = 4 * l;
        const float4 kv = *reinterpret_cast<const float4*>(Ks + row * kLdK + c4);
        const float e = ev[row];
        *reinterpret_cast<float4*>(Qs + row * kLdX + c4) = make_float4(tf32_operand(e * kv.x), tf32_operand(e * kv.y), tf32_operand(e * kv.z), tf32_operand(e * kv.w));
      }
    }
    local_sync();
    invert_unit_lower_64(LT, Tt, Ms);       // ends with a barrier
    // T is lower triangular: row block m needs k < 16 (m + 1).  A warp takes 16 (or 8) columns of two row blocks, (3, 0)
    // or (2, 1), ten k steps either way.
    const int qn = w & 7, m_hi = w < 8 ? 3 : 2, m_lo = w < 8 ? 0 : 1;
    {   // W = T X
      float acc[2][2][4];
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int n = 0; n < 2; ++n) acc[k][n][0] = acc[k][n][1] = acc[k][n][2] = acc[k][n][3] = 0.f;
      warp_gemm_tril_pair<2>(acc[0], acc[1], LT, kLdM, m_hi, m_lo, Qs + qn * 16, kLdX);
      float* dst = ws.WQ + unit * 16384;
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const int col = qn * 16 + n * 8 + 2 * tq, r_lo = (k ? m_lo : m_hi) * 16 + g;
          *reinterpret_cast<float2*>(dst + ((col >> 2) * 128 + r_lo) * 4 + (col & 3)) = make_float2(tf32_operand(acc[k][n][0]), tf32_operand(acc[k][n][1]));
          *reinterpret_cast<float2*>(dst + ((col >> 2) * 128 + r_lo + 8) * 4 + (col & 3)) = make_float2(tf32_operand(acc[k][n][2]), tf32_operand(acc[k][n][3]));
        }
    }
#pragma unroll 1
    for (int round = 0; round < 128 / VCH; ++round) {   // X = beta SiLU(conv(v)) from the staged raw rows, then Ut = T X
      cp_async_wait_all();
      local_sync();                  // the raw rows are there; X = beta e^G K consumed
      constexpr int VP = VCH / 2, VR = 64 / (kLocalThreads / VP);
      const int vch = 2 * (t % VP), vr = (t / VP) * VR;
      f2 v[VR];
      conv_rows<BF16>(a.conv, 2 * KW + h * 128 + round * VCH + vch, RB, VCH, vr, vch, v);
#pragma unroll
      for (int i = 0; i < VR; ++i) {
        const float b = vr + i < valid ? bv[vr + i] : 0.f;
        const float2 x = unpack2(mul2(v[i], pack2(b, b)));
        *reinterpret_cast<float2*>(Qs + (vr + i) * kLdX + round * VCH + vch) = make_float2(tf32_operand(x.x), tf32_operand(x.y));
      }
      local_sync();
      // staging tile consumed: start the next rows
      if (round + 1 < 128 / VCH) stage_issue<BF16, VCH>(P, C, r0, 2 * KW + h * 128 + (round + 1) * VCH, RB);
      else if (vi + 1 < v_last) stage_issue<BF16, VCH>(P, C, r0, 2 * KW + (h + 1) * 128, RB);
      // Ut = T X  (stored fp32: it is added, not multiplied, in the scan)
      constexpr int NT = VCH / 64;
      float acc[2][NT][4];
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int n = 0; n < NT; ++n) acc[k][n][0] = acc[k][n][1] = acc[k][n][2] = acc[k][n][3] = 0.f;
      warp_gemm_tril_pair<NT>(acc[0], acc[1], LT, kLdM, m_hi, m_lo, Qs + round * VCH + qn * NT * 8, kLdX);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int mt2 = k ? m_lo : m_hi;
        // [token / 16][(token % 16) / 4][column][token % 4]: a scan thread owns a column and reads four tokens per
        // 128-bit load, a warp 512 contiguous bytes
        float* dst = ws.Ut + unit * 8192 + (size_t)mt2 * 2048;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const int col = round * VCH + (qn * NT + n) * 8 + 2 * tq;
          float* d = dst + (g >> 2) * 512 + col * 4 + (g & 3);
          d[0] = acc[k][n][0]; d[4] = acc[k][n][1]; d[1024] = acc[k][n][2]; d[1028] = acc[k][n][3];
        }
      }
    }
  }
}

// Units in chunk order: one value head each in the first `split` chunks, one key head with all its value heads after that.
struct LocalUnit { int c, h0, n; };
__device__ __forceinline__ LocalUnit unit_at(int u, int split, int Hv, int Hk) {
  const int rep = Hv / Hk, v = u - split * Hv;
  if (v < 0) return {u / Hv, u % Hv, 1};
  return {split + v / Hk, v % Hk * rep, rep};
}
// grid: CTAs that walk the units, HALVES at a time
template <bool BF16, int HALVES>
__global__ void __launch_bounds__(HALVES * kLocalThreads, 3 - HALVES) gdn_chunk_local_kernel(const __grid_constant__ GdnPrefillParams P, const __grid_constant__ ChunkWs ws, int split) {
  extern __shared__ __align__(16) float sm[];
  const int units = split * P.Hv + (ws.chunks - split) * P.Hk;
  const int step = HALVES * gridDim.x, half = threadIdx.x >> 9, first = blockIdx.x + half * gridDim.x, t = local_tid();
  pdl_wait();
  // The scan, which is let in below, must not see a mark of the call before.  One thread's release counts for the whole CTA, so
  // the first half clears the marks of both and releases alone; the other half meets it (kCleared) before its first mark.
  if (half == 0) {
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
      const LocalUnit x = unit_at(u, split, P.Hv, P.Hk);
      if (t < x.n) ws.ready[(size_t)x.c * P.Hv + x.h0 + t] = 0;
    }
    __threadfence();
    local_sync();
    pdl_release();
    if (HALVES == 2) asm volatile("bar.arrive %0, 1024;\n" ::"n"(kCleared) : "memory");
  }
#pragma unroll 1
  for (int u = first; u < units; u += step) {
    const LocalUnit x = unit_at(u, split, P.Hv, P.Hk);
    const int rep = P.Hv / P.Hk;
    local_unit<BF16>(P, ws, sm + half * (kLocalSmem / sizeof(float)), x.c, x.h0 / rep, x.h0 % rep, x.h0 % rep + x.n);
    asm volatile("fence.proxy.async;\n" ::: "memory");                      // the scan reads the tiles with bulk copies
    if (HALVES == 2 && half == 1 && u == first) asm volatile("bar.sync %0, 1024;\n" ::"n"(kCleared) : "memory");
    local_sync();
    const LocalUnit y = unit_at(u, split, P.Hv, P.Hk);
    if (t < y.n) asm volatile("st.release.gpu.global.u32 [%0], %1;\n" ::"l"(ws.ready + (size_t)y.c * P.Hv + y.h0 + t), "r"(1u) : "memory");
  }
  if (HALVES == 2 && half == 1 && first >= units) asm volatile("bar.sync %0, 1024;\n" ::"n"(kCleared) : "memory");
}

cr_status gdn_chunk_local_launch(const cr_geometry* g, const GdnPrefillParams& P, const ChunkWs& ws, bool bf16_in, cudaStream_t stream) {
  static PerDeviceOnce configured;
  if (cr_status st = once_per_device(configured, [] {
        CR_CUDA(cudaFuncSetAttribute(gdn_chunk_local_kernel<true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLocalSmem));
        CR_CUDA(cudaFuncSetAttribute(gdn_chunk_local_kernel<false, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLocalSmem));
        CR_CUDA(cudaFuncSetAttribute(gdn_chunk_local_kernel<true, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(2 * kLocalSmem)));
        CR_CUDA(cudaFuncSetAttribute(gdn_chunk_local_kernel<false, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(2 * kLocalSmem)));
        return CR_OK;
      })) return st;
  const int Hv = g->gdn_vheads, room = sm_count() - Hv, nch = ws.chunks;
  if (P.chained && room > 0) {
    // The scan follows beside it: one CTA per SM, and an SM left to each of the scan's CTAs.  A short call takes its value heads
    // apart (q and k prepared once per value head) while all units are resident at once.  In a longer one the first halves begin
    // with single heads: the first chunks are ready earlier, and the halves of an SM get out of step (in step, both wait for
    // the same things at the same time; 1,999 rows: 118 us instead of 111 with one half 15 us late).
    const int split = nch * Hv <= 2 * room ? nch : std::min(nch, room / Hv), units = split * Hv + (nch - split) * g->gdn_kheads;
    CR_CUDA(launch_pdl(bf16_in ? gdn_chunk_local_kernel<true, 2> : gdn_chunk_local_kernel<false, 2>, dim3(std::min(units, room)), dim3(2 * kLocalThreads),
                       2 * kLocalSmem, stream, P, ws, split));
    CR_LAUNCH_CHECK("gdn_chunk_local_kernel<2>");        // under a name of its own in stage timing
  } else {
    // A CTA per unit, to run wherever there is room.
    const int split = nch * Hv <= 2 * sm_count() ? nch : 0;
    CR_CUDA(launch_chained(P.chained, bf16_in ? gdn_chunk_local_kernel<true, 1> : gdn_chunk_local_kernel<false, 1>, dim3(split * Hv + (nch - split) * g->gdn_kheads),
                           dim3(kLocalThreads), kLocalSmem, stream, P, ws, split));
    CR_LAUNCH_CHECK("gdn_chunk_local_kernel");
  }
  return CR_OK;
}

}  // namespace cr

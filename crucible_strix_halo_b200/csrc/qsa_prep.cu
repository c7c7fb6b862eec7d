// QSA row preparation for sm_100a: CN-RMSNorm + partial RoPE of the query / key / indexer-query heads, K/V
// rows to the fp16 cache, raw indexer keys, pooled indexer keys of completed 4-token blocks, RoPE table.
// Follows QsaPrepKernel / QsaPoolKernel / QsaRetainRawKernel / QsaPrefillQueryKernel
// (engine/layers/ops.h:561-645; engine/layers/kernels/prefill_qsa.h:35-51, :220-242).
#include "qsa.cuh"

namespace cr {

__global__ void rope_table_kernel(float* table) {
  const int j = threadIdx.x;
  if (j < 32) table[j] = powf(10000000.f, -2.f * j / 64.f);
  else if (j < CR_ROPE_TABLE_FLOATS) table[j] = j == 32 ? 1.f : 0.f;
}

// Cosine and sine of frequency j (< 32) of the row at cache position p.  With a table of multimodal positions (mrope
// [capacity][4]: t, h, w of every cache position; engine/layers/ops.h:515-541) frequency j turns with the h position when
// j % 3 == 1, with the w position when j % 3 == 2 and j < 30, else with t (interleaved sections [11, 11, 10]); equal axes
// give the text rotation exactly.
__device__ __forceinline__ void rope_terms(const cr_qsa_args& a, int j, int p, float& c, float& s) {
  int pj = p;
  if (a.mrope) pj = j % 3 == 1 ? a.mrope[4 * (size_t)p + 1] : (j % 3 == 2 && j < 30 ? a.mrope[4 * (size_t)p + 2] : a.mrope[4 * (size_t)p]);
  rope_cs(a.rope, j, pj, c, s);
}

// Four consecutive floats at p (16-byte aligned where VEC).
template <bool VEC>
__device__ __forceinline__ float4 ld4(const float* p) {
  if constexpr (VEC) return *reinterpret_cast<const float4*>(p);
  else return make_float4(p[0], p[1], p[2], p[3]);
}
template <bool VEC>
__device__ __forceinline__ void st4(float* p, const float4 v) {
  if constexpr (VEC) *reinterpret_cast<float4*>(p) = v;
  else { p[0] = v.x; p[1] = v.y; p[2] = v.z; p[3] = v.w; }
}
template <bool VEC>
__device__ __forceinline__ void st_half4(uint16_t* p, const float4 v) {
  const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
  const unsigned u0 = *reinterpret_cast<const unsigned*>(&lo), u1 = *reinterpret_cast<const unsigned*>(&hi);
  if constexpr (VEC) *reinterpret_cast<uint2*>(p) = make_uint2(u0, u1);
  else { p[0] = (uint16_t)u0; p[1] = (uint16_t)(u0 >> 16); p[2] = (uint16_t)u1; p[3] = (uint16_t)(u1 >> 16); }
}

// A head of 256 values spread over a warp: lane l holds elements 4 l .. 4 l + 3 and 128 + 4 l .. + 3.
// CN-RMSNorm, then split-half RoPE of the first 64: lanes 0-7 hold the first half of the pairs, lanes 8-15 the second.
// c4 / s4: cosines and sines of the frequencies 4 (l % 8) .. + 3.
template <bool VEC>
__device__ __forceinline__ void norm_rope(float4 (&x)[2], const float* w1, const float4 c4, const float4 s4) {
  const int l = threadIdx.x & 31;
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < 2; ++i) ss += x[i].x * x[i].x + x[i].y * x[i].y + x[i].z * x[i].z + x[i].w * x[i].w;
  const float rs = rsqrtf(warp_sum(ss) / 256.f + kEps);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float4 w = ld4<VEC>(w1 + 128 * i + 4 * l);
    x[i] = make_float4(x[i].x * rs * w.x, x[i].y * rs * w.y, x[i].z * rs * w.z, x[i].w * rs * w.w);
  }
  float4 o;                                              // the partner of every element: j and j + 32
  o.x = __shfl_xor_sync(0xffffffffu, x[0].x, 8); o.y = __shfl_xor_sync(0xffffffffu, x[0].y, 8);
  o.z = __shfl_xor_sync(0xffffffffu, x[0].z, 8); o.w = __shfl_xor_sync(0xffffffffu, x[0].w, 8);
  if (l < 16) {
    const float sg = l < 8 ? -1.f : 1.f;
    x[0] = make_float4(x[0].x * c4.x + sg * o.x * s4.x, x[0].y * c4.y + sg * o.y * s4.y, x[0].z * c4.z + sg * o.z * s4.z,
                       x[0].w * c4.w + sg * o.w * s4.w);
  }
}

// A head of the indexer (128 values), strided over a warp: lane l holds the elements l, 32 + l, 64 + l, 96 + l.  The sum of
// squares is the left-to-right sum of the four 32-element butterflies: selections hang on the last bit of these rows, so
// the order of the additions stays what it is.  cj / sj: cosine and sine of frequency l.
__device__ __forceinline__ void norm_rope_idx(float (&x)[4], const float* w1, float cj, float sj) {
  const int l = threadIdx.x & 31;
  float t[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) t[i] = warp_sum(x[i] * x[i]);
  const float rs = rsqrtf((((t[0] + t[1]) + t[2]) + t[3]) / 128.f + kEps);
#pragma unroll
  for (int i = 0; i < 4; ++i) x[i] = x[i] * rs * w1[32 * i + l];
  const float a = x[0], b = x[1];
  x[0] = a * cj - b * sj;
  x[1] = b * cj + a * sj;
}

// Rows at which a call keeps only the newest raw keys of a ring (a longer call writes the ring once, at its end).
__device__ __forceinline__ bool raw_kept(const cr_qsa_args& a, int r) { return a.c.raw_slots == 0 || r >= a.R - a.c.raw_slots; }
// Whether the ring slot of row r is that of one of the positions before this call that share the call's first block:
// the warp that pools the block reads them first and writes those rows itself.
__device__ __forceinline__ bool raw_after_pool(const cr_qsa_args& a, int r) {
  if (a.c.raw_slots == 0 || a.pos0 % 4 == 0 || (a.pos0 + a.R) / 4 == a.pos0 / 4) return false;
  for (int p = a.pos0 / 4 * 4; p < a.pos0; ++p)
    if ((a.pos0 + r - p) % a.c.raw_slots == 0) return true;
  return false;
}

// Pooled key of block b (complete within rows pos0..pos0+R-1 or earlier) by one warp: mean of 4 raw keys -> fp16 round ->
// CN-RMSNorm -> RoPE at the block start.  Raw keys of this call's rows are read from the input rows, older ones from the
// cache, so the result does not depend on the other warps having run.
template <bool VEC>
__device__ __forceinline__ void pool_block(const cr_qsa_args& a, int b) {
  const int l = threadIdx.x & 31;
  float k[4][4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int pos = b * 4 + t;
    const float* src = pos >= a.pos0 ? a.idx + (size_t)(pos - a.pos0) * 640 + 512 + l : a.c.ik_raw + raw_offset(a.c.raw_slots, pos, l);
#pragma unroll
    for (int i = 0; i < 4; ++i) k[t][i] = src[32 * i];
  }
  float cj, sj, x[4];
  rope_terms(a, l, b * 4, cj, sj);
#pragma unroll
  for (int i = 0; i < 4; ++i) x[i] = round_h((((k[0][i] + k[1][i]) + k[2][i]) + k[3][i]) * 0.25f);
  norm_rope_idx(x, a.ik_norm1, cj, sj);
#pragma unroll
  for (int i = 0; i < 4; ++i) a.c.ik_pool[pool_offset(b, 32 * i + l)] = x[i];
  if (b == a.pos0 / 4 && a.c.raw_slots != 0) {            // the ring rows that had to wait for the reads above
    __syncwarp();
    for (int r0 = max(0, a.R - a.c.raw_slots); r0 < a.R; r0 += 32) {       // a lane looks at a row: at most three have to be written
      unsigned rows = __ballot_sync(0xffffffffu, r0 + l < a.R && raw_after_pool(a, r0 + l));
      for (; rows; rows &= rows - 1) {
        const int r = r0 + __ffs(rows) - 1;
        st4<VEC>(a.c.ik_raw + raw_offset(a.c.raw_slots, a.pos0 + r, 4 * l), ld4<VEC>(a.idx + (size_t)r * 640 + 512 + 4 * l));
      }
    }
  }
}

// grid (unit groups, Rmax, spans), 256 threads; a warp takes the units blockIdx.x * 8 * UPW + w + 8 i, i < UPW, of one row.
// Units: [0, Hq) query heads, [.., + Hkv) key heads, [.., + Hkv) value heads, 4 indexer-query heads, the raw indexer key, and
// the pooled key of the block that the row completes.  u0 skips leading units (u0 = Hq runs the cache units only).
// q_hi (optional): fp16 copy of the prepared queries [R][Hq][256] for the prefill attention kernels; rows < q_skip are
// not written to q_hi.  mark_dense: rows that attend every block say so here (nsel = -1), which saves a call of such rows
// alone the launch of the selection.  queries_only: only the query and indexer-query units do anything (a rank of a split-KV group that
// does not own the rows' positions still normalises the queries).
//
// Bound: HBM for a part (query rows in and out, fp16 copies, cache rows), latency for a step.  A head lives in one warp
// (128-bit loads, shuffle reduction, no barrier but the one behind the row's 32 cosines and sines, which every unit of the
// row shares).  A step gives every unit a warp of its own (UPW = 1); a part
// takes a row per CTA with all loads of a warp issued first (UPW = 5).  2,048 rows at 262,144 positions: 98.8 us as one
// CTA per (row, unit), 28 us now (4.9 TB/s).  With a compact ring the warp that pools a call's first block looked at sixteen rows one by
// one, two divisions for each of three positions: 10.0 us for 117 rows where a full raw cache took 3.9; a lane per row now.
template <int UPW, bool VEC>
__global__ void __launch_bounds__(256) qsa_prep_kernel(const __grid_constant__ QsaParams P, int u0, __half* q_hi, int q_skip, int queries_only, int mark_dense) {
  pdl_release();
  pdl_wait();
  const cr_qsa_args& a = P.span[blockIdx.z];
  const int r = blockIdx.y;
  if (r >= a.R) return;
  __shared__ __align__(16) float cs[32], sn[32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, p = a.pos0 + r, Hq = P.Hq, Hkv = P.Hkv;
  const int first = u0 + blockIdx.x * 8 * UPW + w;
  float4 x[UPW][2];
#pragma unroll
  for (int i = 0; i < UPW; ++i) {
    const int u = first + 8 * i;
    const float* src = nullptr;
    bool wide = true;
    if (u < Hq) src = a.q + ((size_t)r * Hq + u) * 512;
    else if (u < Hq + 2 * Hkv) src = queries_only ? nullptr : (u < Hq + Hkv ? a.k + ((size_t)r * Hkv + u - Hq) * 256 : a.v + ((size_t)r * Hkv + u - Hq - Hkv) * 256);
    else if (u < Hq + 2 * Hkv + 5) { src = u < Hq + 2 * Hkv + 4 || !queries_only ? a.idx + (size_t)r * 640 + (u - Hq - 2 * Hkv) * 128 : nullptr; wide = false; }
    x[i][0] = x[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (src) {
      if (wide) { x[i][0] = ld4<VEC>(src + 4 * l); x[i][1] = ld4<VEC>(src + 128 + 4 * l); }
      else x[i][0] = make_float4(src[l], src[32 + l], src[64 + l], src[96 + l]);
    }
  }
  if (w == 0) {
    float c, s;
    rope_terms(a, l, p, c, s);
    cs[l] = c; sn[l] = s;
  }
  __syncthreads();
  const float4 c4 = *reinterpret_cast<const float4*>(&cs[4 * (l & 7)]), s4 = *reinterpret_cast<const float4*>(&sn[4 * (l & 7)]);
#pragma unroll
  for (int i = 0; i < UPW; ++i) {
    const int u = first + 8 * i;
    if (u < Hq) {
      norm_rope<VEC>(x[i], a.q_norm1, c4, s4);
      float* q = a.q + ((size_t)r * Hq + u) * 512 + 4 * l;
      st4<VEC>(q, x[i][0]);
      st4<VEC>(q + 128, x[i][1]);
      if (q_hi && r >= q_skip) {
        uint16_t* h = reinterpret_cast<uint16_t*>(q_hi) + ((size_t)r * Hq + u) * 256 + 4 * l;
        st_half4<VEC>(h, x[i][0]);
        st_half4<VEC>(h + 128, x[i][1]);
      }
    } else if (u < Hq + 2 * Hkv) {
      if (queries_only) continue;
      const bool key = u < Hq + Hkv;
      if (key) norm_rope<VEC>(x[i], a.k_norm1, c4, s4);
      uint16_t* h = (key ? a.c.k : a.c.v) + ((size_t)p * Hkv + (u - Hq - (key ? 0 : Hkv))) * 256 + 4 * l;
      st_half4<VEC>(h, x[i][0]);
      st_half4<VEC>(h + 128, x[i][1]);
    } else if (u < Hq + 2 * Hkv + 4) {
      float y[4] = {x[i][0].x, x[i][0].y, x[i][0].z, x[i][0].w};
      norm_rope_idx(y, a.iq_norm1, cs[l], sn[l]);
      float* dst = a.idx + (size_t)r * 640 + (u - Hq - 2 * Hkv) * 128 + l;
      dst[0] = y[0]; dst[32] = y[1]; dst[64] = y[2]; dst[96] = y[3];
    } else if (queries_only) {
      continue;
    } else if (u == Hq + 2 * Hkv + 4) {
      if (mark_dense && l == 0 && (p + 1) / 4 <= CR_SEL_BLOCKS) a.nsel[r] = -1;
      if (raw_kept(a, r) && !raw_after_pool(a, r)) {
        float* dst = a.c.ik_raw + raw_offset(a.c.raw_slots, p, l);
        dst[0] = x[i][0].x; dst[32] = x[i][0].y; dst[64] = x[i][0].z; dst[96] = x[i][0].w;
      }
    } else if (u == Hq + 2 * Hkv + 5) {
      if (p % 4 == 3) pool_block<VEC>(a, p / 4);
    }
  }
}

cr_status qsa_validate(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, int max_rows, const char* who, int score_blocks) {
  if (cr_status s = check_geometry(g)) return s;
  CR_REQUIRE(spans && n_spans >= 1, "%s: no spans", who);
  for (int s = 0; s < n_spans; ++s) {
    const cr_qsa_args& a = spans[s];
    CR_REQUIRE(a.R >= 1 && a.R <= max_rows, "%s: span %d has R=%d, need 1..%d", who, s, a.R, max_rows);
    CR_REQUIRE(a.pos0 >= 0, "%s: span %d has negative pos0", who, s);
    const int need_stride = score_blocks >= 0 ? score_blocks : (a.pos0 + a.R) / 4;   // entries that score a block range need that range only
    CR_REQUIRE(a.sstride >= need_stride, "%s: span %d score stride %d < %d blocks", who, s, a.sstride, need_stride);
    CR_REQUIRE(a.q && a.k && a.v && a.idx && a.q_norm1 && a.k_norm1 && a.iq_norm1 && a.ik_norm1 && a.c.k && a.c.v &&
               a.c.ik_raw && a.c.ik_pool && a.sel && a.nsel && a.rope, "%s: span %d has a null buffer", who, s);
    CR_REQUIRE(a.scores || (a.pos0 + a.R) / 4 <= CR_SEL_BLOCKS, "%s: span %d needs a score buffer", who, s);
    CR_REQUIRE(a.c.raw_slots == 0 || a.c.raw_slots >= 16, "%s: span %d raw ring of %d slots is too small", who, s, a.c.raw_slots);
  }
  return CR_OK;
}

int qsa_max_rows(const cr_qsa_args* spans, int n) {
  int m = 0;
  for (int s = 0; s < n; ++s) m = spans[s].R > m ? spans[s].R : m;
  return m;
}

void qsa_fill_params(QsaParams& P, const cr_geometry* g, const cr_qsa_args* spans, int n) {
  for (int s = 0; s < n; ++s) P.span[s] = spans[s];
  int base = 0;
  for (int s = 0; s < n; ++s) { P.base[s] = base; base += spans[s].R; }
  P.Hq = g->q_heads; P.Hkv = g->kv_heads; P.n = n;
  P.b_lo = 0; P.b_hi = INT_MAX;
  P.tile_count = nullptr; P.tile_rows = 1; P.tile_max = 0; P.tile_mixed = -1;
}

cr_status qsa_prep_launch(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, int u0, __half* q_hi, int q_skip,
                          cudaStream_t stream, bool queries_only, bool mark_dense) {
  use_stream(stream);
  for (int s0 = 0; s0 < n_spans; s0 += kMaxSpans) {
    const int n = n_spans - s0 < kMaxSpans ? n_spans - s0 : kMaxSpans;
    QsaParams P;
    qsa_fill_params(P, g, spans + s0, n);
    const int Rmax = qsa_max_rows(spans + s0, n);
    const int units = g->q_heads + 2 * g->kv_heads + 6 - u0;
    bool vec = ((uintptr_t)q_hi & 7) == 0;          // buffers at 4-byte boundaries take scalar accesses
    for (int s = 0; s < n && vec; ++s) {
      const cr_qsa_args& a = spans[s0 + s];
      for (const void* ptr : {(const void*)a.q, (const void*)a.k, (const void*)a.v, (const void*)a.idx, (const void*)a.q_norm1, (const void*)a.k_norm1,
                              (const void*)a.iq_norm1, (const void*)a.ik_norm1, (const void*)a.c.k, (const void*)a.c.v, (const void*)a.c.ik_raw})
        vec = vec && ((uintptr_t)ptr & 15) == 0;
    }
    constexpr int kBulk = 5;                       // 40 units: every row of the built geometries in one CTA
    const bool bulk = (long long)Rmax * n > 128;    // below that a CTA per row would leave SMs idle
    auto kernel = bulk ? (vec ? qsa_prep_kernel<kBulk, true> : qsa_prep_kernel<kBulk, false>) : (vec ? qsa_prep_kernel<1, true> : qsa_prep_kernel<1, false>);
    const int per_cta = 8 * (bulk ? kBulk : 1);
    CR_CUDA(launch_pdl(kernel, dim3((units + per_cta - 1) / per_cta, Rmax, n), dim3(256), 0, stream, P, u0, q_hi, q_skip, queries_only ? 1 : 0, mark_dense ? 1 : 0));
    CR_LAUNCH_CHECK("qsa_prep_kernel");
  }
  return CR_OK;
}

}  // namespace cr

extern "C" cr_status cr_rope_table_fill(float* table, void* stream) {
  using namespace cr;
  CR_REQUIRE(table, "cr_rope_table_fill: null table");
  use_stream((cudaStream_t)stream);
  rope_table_kernel<<<1, CR_ROPE_TABLE_FLOATS, 0, (cudaStream_t)stream>>>(table);
  CR_LAUNCH_CHECK("rope_table_kernel");
  return CR_OK;
}

// YaRN table for a context of factor x 262,144 positions (the rows of engine/layers/rope_tables.h; Hugging Face
// "yarn" rope scaling with original context 262,144, beta_fast 32, beta_slow 1, rotary dim 64, theta 1e7): frequencies
// that turn more than 32 times over the original context are kept, those that turn less than once are divided by the
// factor, a linear ramp in between; the cos/sin multiplier is 0.1 ln(factor) + 1.
extern "C" cr_status cr_rope_table_fill_yarn(float* table, int factor, void* stream) {
  using namespace cr;
  CR_REQUIRE(table, "cr_rope_table_fill_yarn: null table");
  CR_REQUIRE(factor >= 1 && factor <= 64, "cr_rope_table_fill_yarn: factor %d outside 1..64", factor);
  if (factor == 1) return cr_rope_table_fill(table, stream);
  constexpr double kDim = 64.0, kBase = 1e7, kOrig = 262144.0, kPi = 3.14159265358979323846;
  auto turns_dim = [&](double turns) { return kDim * log(kOrig / (turns * 2.0 * kPi)) / (2.0 * log(kBase)); };
  double low = floor(turns_dim(32.0)), high = ceil(turns_dim(1.0));
  low = low < 0 ? 0 : low;
  high = high > kDim - 1 ? kDim - 1 : high;
  if (low == high) high += 0.001;
  float host[CR_ROPE_TABLE_FLOATS] = {};
  for (int j = 0; j < 32; ++j) {
    const float extrap = 1.0f / powf(10000000.f, (float)(2 * j) / 64.f), interp = extrap / (float)factor;
    float ramp = ((float)j - (float)low) / ((float)high - (float)low);
    ramp = ramp < 0.f ? 0.f : (ramp > 1.f ? 1.f : ramp);
    const float keep = 1.f - ramp;                        // share of the original frequency
    host[j] = interp * (1.f - keep) + extrap * keep;
  }
  host[32] = (float)(0.1 * log((double)factor) + 1.0);
  CR_CUDA(cudaMemcpyAsync(table, host, sizeof(host), cudaMemcpyHostToDevice, (cudaStream_t)stream));   // pageable source: staged before the call returns
  return CR_OK;
}

// The query units of cr_qsa_prep alone: q heads and indexer-query heads normalised + roped in place; no cache row, raw
// key or pooled key is written.  For the ranks of a split-KV group that do not own the rows' positions.  No counterpart
// in the single-device reference.
extern "C" cr_status cr_qsa_prep_queries(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, void* stream) {
  using namespace cr;
  if (cr_status s = qsa_validate(g, spans, n_spans, CR_MAX_PREFILL_ROWS, "cr_qsa_prep_queries", 0)) return s;
  return qsa_prep_launch(g, spans, n_spans, 0, nullptr, 0, (cudaStream_t)stream, true);
}

extern "C" cr_status cr_qsa_prep(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, void* stream) {
  using namespace cr;
  if (cr_status s = qsa_validate(g, spans, n_spans, CR_MAX_STEP_ROWS, "cr_qsa_prep")) return s;
  return qsa_prep_launch(g, spans, n_spans, 0, nullptr, 0, (cudaStream_t)stream);
}

extern "C" cr_status cr_qsa_prefill_cache(const cr_geometry* g, const cr_qsa_args* a, void* stream) {
  using namespace cr;
  if (cr_status s = qsa_validate(g, a, 1, CR_MAX_PREFILL_ROWS, "cr_qsa_prefill_cache")) return s;
  return qsa_prep_launch(g, a, 1, g->q_heads, nullptr, 0, (cudaStream_t)stream);
}

extern "C" size_t cr_qsa_pool_floats(int ctx) { return (size_t)((ctx + 127) / 128) * 4096; }

extern "C" cr_status cr_qsa_cache_bytes(const cr_geometry* g, int ctx, int bounded, size_t out_bytes[4]) {
  using namespace cr;
  if (cr_status s = check_geometry(g)) return s;
  CR_REQUIRE(out_bytes, "cr_qsa_cache_bytes: null output");
  CR_REQUIRE(ctx >= 1 && ctx <= 1048576, "cr_qsa_cache_bytes: context %d is out of range", ctx);
  out_bytes[0] = out_bytes[1] = (size_t)ctx * g->kv_heads * 256 * 2;
  out_bytes[2] = (size_t)(bounded ? 16 : ctx) * 128 * sizeof(float);
  out_bytes[3] = cr_qsa_pool_floats(ctx) * sizeof(float);
  return CR_OK;
}

// Shared declarations of the QSA kernels (qsa_prep.cu, qsa_select.cu, qsa_attn.cu, qsa_prefill.cu).
#pragma once
#include <climits>
#include "common.cuh"

namespace cr {

// All spans of one launch; base[s] = first row of span s in scratch laid out by row.
struct QsaParams {
  cr_qsa_args span[kMaxSpans];
  int base[kMaxSpans];
  int Hq, Hkv, n;
  int b_lo, b_hi;          // scoring only: the blocks [b_lo, b_hi) are scored (a rank's own blocks; 0, INT_MAX = all)
  // Prefill parts whose rows go to the tiled or to the row-wise attention by their union lists (null: all row-wise).
  const int* tile_count;   // entries of every tile's list
  int tile_rows, tile_max; // rows of a tile; entries per row up to which the tiled kernel is the quicker one
  int tile_mixed;          // >= 0: one decision for the whole part, with this line where some tile has to go row-wise all the same
};
// Tiles of more entries per row than this go row-wise whatever their part does: they would gain little, and the row-wise kernel
// splits queries and probabilities into two fp16 numbers where the tiled one rounds them to one.
constexpr int kTileMost = 298;
// Which kernel serves the rows of `tile`: true, the tiled one.  Called by whole warps.  rows: rows of the part, of which the last tile
// may hold fewer than tile_rows.
__device__ __forceinline__ bool qsa_tile_shares(const int* count, int tile, int tile_rows, int rows, int per_row, int mixed) {
  if (per_row >= CR_SEL_BLOCKS + 1) return true;         // no list is longer
  const int here = min(tile_rows, rows - tile * tile_rows), entries = count[tile];
  if (mixed >= 0) {
    int sum = 0;
    bool over = false;
    for (int i = threadIdx.x & 31; i * tile_rows < rows; i += 32) {
      const int n = count[i];
      sum += n;
      over |= n > kTileMost * min(tile_rows, rows - i * tile_rows);
    }
    const int line = __any_sync(0xffffffffu, over) ? mixed : per_row;
    return ((int)__reduce_add_sync(0xffffffffu, sum) <= line * rows) & (entries <= kTileMost * here);
  }
  // A last tile of few rows has few entries and many per row: it follows the tile before it.
  const bool ragged = here < tile_rows && tile > 0;
  const int decides = ragged ? count[tile - 1] : entries;
  return (entries <= kTileMost * here) & (decides <= per_row * (tile > 0 ? tile_rows : here));
}
__device__ __forceinline__ bool qsa_row_is_tiled(const QsaParams& P, int r) {
  return P.tile_count && qsa_tile_shares(P.tile_count, r / P.tile_rows, P.tile_rows, P.span[0].R, P.tile_max, P.tile_mixed);
}

// score_blocks >= 0: the score stride must cover that many blocks (a rank's own range, or 0 for entries that never touch
// the scores) instead of every block of the rows.
cr_status qsa_validate(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, int max_rows, const char* who, int score_blocks = -1);
int qsa_max_rows(const cr_qsa_args* spans, int n);
void qsa_fill_params(QsaParams& P, const cr_geometry* g, const cr_qsa_args* spans, int n);
cr_status qsa_prep_launch(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, int u0, __half* q_hi, int q_skip,
                          cudaStream_t stream, bool queries_only = false, bool mark_dense = false);
cr_status qsa_score_launch(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, cudaStream_t stream, int b_lo = 0, int b_hi = INT_MAX);
// Prefill parts (many rows): the scores as four GEMMs on tcgen05 tensor cores.
cr_status qsa_score_tc_launch(const QsaParams& P, int n, cudaStream_t stream);
// Spans of 3..16 rows (verify passes): the scores as an HBM stream through mma.sync, every block of every row.
// wide: every pool lies at a 16-byte boundary.
cr_status qsa_score_mma_launch(const QsaParams& P, int tiles, int Rmax, int n, bool wide, cudaStream_t stream);
cr_status qsa_topk_launch(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, cudaStream_t stream, bool dense_marked = false);
cr_status qsa_select_launch(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, cudaStream_t stream, bool dense_marked = false);
struct QsaTileSplit { const int* count; int rows, max, mixed; };   // see QsaParams::tile_count
// Attention of the spans' rows over the attended positions inside [p0, p1): outputs, or with `partials` one (m, l, acc[256])
// record per (row, head).
cr_status qsa_attn_launch(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, float* partials, int p0, int p1, cr_out_format fmt,
                          cudaStream_t stream, const QsaTileSplit* tiles = nullptr);

// Combines `nparts` (at most 32) records per (row, head), record p of row r at partials[(p * R + r) * Hq + h], into outputs;
// with `tiles` only the rows of tiled tiles have records.
cr_status qsa_merge_launch(const cr_geometry* g, const cr_qsa_args& a, int nparts, const float* partials, cr_out_format fmt, cudaStream_t stream,
                           const QsaTileSplit* tiles = nullptr);

// Channels c .. c + 3 (c = 128 half + 4 lane, a warp holds a 128-channel group) of one head of one row: un-gated context,
// gate, output format.
__device__ __forceinline__ void emit_group(const cr_qsa_args& a, int Hq, int r, int h, int c, float4 o, const float4 gate, int fmt) {
  const size_t W = (size_t)Hq * 256, at = (size_t)r * W + h * 256 + c;
  if (a.context) { float* cx = a.context + at; cx[0] = o.x; cx[1] = o.y; cx[2] = o.z; cx[3] = o.w; }
  float v[4] = {o.x * sigmoidf_(gate.x), o.y * sigmoidf_(gate.y), o.z * sigmoidf_(gate.z), o.w * sigmoidf_(gate.w)};
  if (fmt == CR_OUT_RAW_F32) {
    float* dst = reinterpret_cast<float*>(a.out) + at;
    if (((uintptr_t)dst & 15) == 0) *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
    else { dst[0] = v[0]; dst[1] = v[1]; dst[2] = v[2]; dst[3] = v[3]; }
  } else if (fmt == CR_OUT_RAW_BF16) {
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(a.out) + at;
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
    if (((uintptr_t)dst & 7) == 0) *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
    else { dst[0] = lo.x; dst[1] = lo.y; dst[2] = hi.x; dst[3] = hi.y; }
  } else {
    float su[4];
    load_half4(a.suh_o + h * 256 + c, su);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = round_h(round_h(v[i]) * su[i]);
    wht128(v);
    store_half4(reinterpret_cast<uint16_t*>(a.out) + out_index(r, h * 256 + c, (int)W, a.pack_rows, a.pack_off), v, kHadNorm);   // c is a multiple of 4
  }
}

}  // namespace cr

// QSA prefill part (1..2048 rows against the growing cache) for sm_100a: cache rows, query prep, scores,
// selection, attention with the fused gate.  Entry point of a part, in the role of LaunchQsaPrefillUnion /
// LaunchQsaPrefill (engine/layers/kernels/prefill_qsa_union.h:782-807; prefill_qsa.h:274-299).
// Attention runs over row tiles on tcgen05 tensor cores (qsa_flash.cu: union lists + masked flash attention); the
// row-wise kernel of the decode path (qsa_attn.cu) serves the tiles whose rows share little, and every row with
// cr_options.qsa_union_rows = -1.  Rows of a part are independent once the cache and the pool hold the
// part, so causality inside the part falls out of pos0 + r.
#include <algorithm>
#include <climits>
#include "qsa.cuh"

namespace cr {
int qsa_union_rows(const cr_geometry* g);
int qsa_union_cap(int RT);
cr_status qsa_union_build_launch(const cr_geometry* g, const cr_qsa_args& a, int2* list, int* count, cudaStream_t stream);
cr_status qsa_flash_launch(const cr_geometry* g, const cr_qsa_args& a, const __half* q_hi, const int2* list, const int* count,
                           float* partials, int splits, cr_out_format fmt, int flash_max, int flash_mixed, cudaStream_t stream);

// Scratch of a part: [partial records of split tiles][union lists, 2 ints per entry][union counts].  The list area is sized for tiles of 8 rows, the smallest tile.
//
// A short part has fewer (tile, KV head) pairs than the GPU has SMs, and each walks its whole union list: its tiles are
// then split along the list, as many ways as fill the SMs once, and a merge kernel combines the records.  117 rows at
// 9,003 positions (16 CTAs): 221 us unsplit, 32 us in 9 splits plus 5 us of merge.
constexpr int kMaxTileSplits = 16, kPartialRows = 16 * 160;
static int tile_splits(const cr_geometry* g, int rows) {
  const int RT = qsa_union_rows(g), ctas = (rows + RT - 1) / RT * g->kv_heads, s = sm_count() / ctas;
  const int most = kPartialRows / rows < kMaxTileSplits ? kPartialRows / rows : kMaxTileSplits;
  return s < 1 ? 1 : (s > most ? most : s);
}
// At most kPartialRows rows x splits; grows with the rows, so that the scratch of a long part serves every shorter one.
static size_t partial_bytes(const cr_geometry* g, int rows) {
  const int all = rows * kMaxTileSplits;
  return (size_t)(all < kPartialRows ? all : kPartialRows) * g->q_heads * CR_QSA_PART * sizeof(float);
}
static size_t list_ints(int rows) { return (size_t)((rows + 7) / 8) * qsa_union_cap(8) * 2; }
// Which of the two kernels serves a part, or a tile of it.  Measured on parts of 2 to 2,048 rows at 8 K to 262 K positions, where the
// position hardly matters (sparse rows, us of the attention stage):
//   row-wise, up to 8 heads per KV head   4 + 24 for each wave of one (row, KV head) per SM: 28 to 74 rows, 50 to 54 to 148, 188 at 512,
//                                         660 at 2,048;
//   row-wise, 9 to 12 heads (two warps)   19.5 to 16 rows, 31 to 37, then 53 per wave: 53 to 74 rows, 112 to 148, 1,490 at 2,048;
//   tiled                                 29 + 1.1 for each entry of a row (of 16 in a tile) and wave of CTAs, divided by the splits of a list:
//                                         128 rows of 16 heads 30 at 42 entries and 64 at 264, 1,024 rows 76 and 318, 2,048 rows 142
//                                         and 626.
// The lines below stand where the kernels crossed while the tiled one took 24 + 1.3 (2,048 rows 150 and 700).  Since then they cross later, at 283
// entries for 243 at 2,048 rows and at 250 for 213 at 768; the tiles between the two stay row-wise, with the bits that it keeps of queries and
// probabilities.
// Two warps: the tiled kernel from 17 rows on, whatever the rows share.  (Rows that share little cross later, 17 to 37 rows at 200 entries a
// row, where they take 31 us row-wise and 33 to 40 tiled above that, 64 to 74 rows at 340, 128 rows beyond 513.)
// One warp: a part of one wave row-wise (64 rows at 42 entries, nearly the fewest: 27 to 29 tiled).  Above that the lists decide.
// While every tile has an SM of its own, a tile left out makes the tiled kernel no quicker and the row-wise launch beside it costs
// its whole waves (192 rows about the line, tile by tile: 108 us, either kernel alone 81 to 86), so the part goes one way; lists
// built in vain cost 12 us at 117 rows and 23 at 512, and a wave of row-wise CTAs for a tile past kTileMost 30.  With the lists paid for
// the lines cross at 263 entries per row for 128 and 512 rows, 213 for 768 (one CTA per tile).  Longer parts decide tile by tile:
// 165 entries for 1,204 rows, 243 for 2,048, two waves of CTAs either way.
static bool one_warp_streams(const cr_geometry* g) { return g->q_heads / g->kv_heads <= 8; }
static bool rows_go_row_wise(const cr_geometry* g, int rows) { return one_warp_streams(g) ? rows * g->kv_heads <= sm_count() : rows <= 16; }
static QsaTileSplit tile_rule(const cr_geometry* g, int rows, const int* count, int RT) {
  if (!one_warp_streams(g)) return {count, RT, CR_SEL_BLOCKS + 1, -1};
  auto waves = [](int n) { return (n + sm_count() - 1) / sm_count(); };
  const bool whole = (rows + RT - 1) / RT * g->kv_heads <= sm_count();
  const double per_entry = 1.3 * RT / 16 * waves(std::max(rows / RT, 1) * g->kv_heads) / tile_splits(g, rows);   // a ragged last tile is short
  const double row_wise = 5 + 24.0 * waves(rows * g->kv_heads), vain = 12 + 0.03 * rows;
  auto line = [&](double more) { return std::max(std::min((int)((row_wise - 24 + more) / per_entry), kTileMost), 0); };
  return {count, RT, line(whole ? vain : -2), whole ? line(vain - 30) : -1};
}

static cr_status check_part(const cr_geometry* g, const cr_qsa_prefill_args* args, int skip, cr_out_format fmt, const char* who) {
  CR_REQUIRE(args, "%s: null args", who);
  if (cr_status s = qsa_validate(g, &args->input, 1, CR_MAX_PREFILL_ROWS, who)) return s;
  const cr_qsa_args& q = args->input;
  CR_REQUIRE(skip >= 0 && skip < q.R && skip % 16 == 0, "%s: skip=%d must be a multiple of 16 below R=%d", who, skip, q.R);
  CR_REQUIRE(fmt == CR_OUT_RAW_F32 || fmt == CR_OUT_RAW_BF16 || fmt == CR_OUT_EXL3_WHT, "%s: bad output format", who);
  CR_REQUIRE(q.out && (fmt != CR_OUT_EXL3_WHT || q.suh_o), "%s: output buffer (and suh_o for the EXL3 output) needed", who);
  CR_REQUIRE(fmt == CR_OUT_EXL3_WHT || q.pack_rows == 0, "%s: packed layout only with the EXL3 output", who);
  const size_t need = cr_qsa_prefill_scratch_bytes(g, q.R - skip);
  CR_REQUIRE(args->scratch && args->scratch_bytes >= need, "%s: scratch of %zu bytes needed, %zu given", who, need, args->scratch_bytes);
  CR_REQUIRE(((uintptr_t)args->scratch & 15) == 0, "%s: scratch must be 16-byte aligned", who);
  return CR_OK;
}

// The rows [skip, R) of a part as an argument block of their own.
static cr_qsa_args output_rows(const cr_geometry* g, cr_qsa_args q, int skip, cr_out_format fmt) {
  const size_t W = (size_t)g->q_heads * 256;
  q.pos0 += skip; q.R -= skip;
  q.q += (size_t)skip * g->q_heads * 512; q.idx += (size_t)skip * 640;
  if (q.context) q.context += (size_t)skip * W;
  if (q.pack_rows) q.pack_off += skip;
  else q.out = (char*)q.out + (size_t)skip * W * (fmt == CR_OUT_RAW_F32 ? 4 : 2);
  return q;
}

// Attention of the output rows with sel / nsel in place.
static cr_status attend(const cr_geometry* g, const cr_qsa_prefill_args* args, const cr_qsa_args& q, int skip, cr_out_format fmt,
                        cudaStream_t stream) {
  char* scratch = (char*)args->scratch;
  if (args->q_hi && (options().qsa_union_rows > 0 || (options().qsa_union_rows == 0 && !rows_go_row_wise(g, q.R)))) {
    int2* list = reinterpret_cast<int2*>(scratch + partial_bytes(g, q.R));
    int* count = reinterpret_cast<int*>(list + list_ints(q.R) / 2);
    const int RT = qsa_union_rows(g);
    const int splits = tile_splits(g, q.R);
    QsaTileSplit tiles = tile_rule(g, q.R, count, RT);
    if (options().qsa_union_rows > 0) tiles.max = CR_SEL_BLOCKS + 1;   // an explicit tile size forces the tiled kernel
    if (cr_status s = qsa_union_build_launch(g, q, list, count, stream)) return s;
    if (cr_status s = qsa_flash_launch(g, q, reinterpret_cast<const __half*>(args->q_hi) + (size_t)skip * g->q_heads * 256, list, count,
                                       reinterpret_cast<float*>(scratch), splits, fmt, tiles.max, tiles.mixed, stream)) return s;
    if (splits > 1)
      if (cr_status s = qsa_merge_launch(g, q, splits, reinterpret_cast<const float*>(scratch), fmt, stream, &tiles)) return s;
    if (tiles.max > CR_SEL_BLOCKS) return CR_OK;       // no list is longer
    // the tiles with little sharing: row-wise attention (its CTAs of tiled rows exit at once)
    return qsa_attn_launch(g, &q, 1, nullptr, 0, INT_MAX, fmt, stream, &tiles);
  }
  return qsa_attn_launch(g, &q, 1, nullptr, 0, INT_MAX, fmt, stream);
}
}  // namespace cr

extern "C" size_t cr_qsa_prefill_scratch_bytes(const cr_geometry* g, int rows) {
  if (!g || rows < 1) return 0;
  return cr::partial_bytes(g, rows) + cr::list_ints(rows) * sizeof(int) + (size_t)((rows + 7) / 8) * sizeof(int);
}

extern "C" size_t cr_qsa_union_list_ints(const cr_geometry* g, int rows) {
  if (!g || rows < 1 || cr::check_geometry(g) != CR_OK) return 0;
  const int RT = cr::qsa_union_rows(g);
  return (size_t)((rows + RT - 1) / RT) * cr::qsa_union_cap(RT) * 2;
}

extern "C" int cr_qsa_union_tile_rows(const cr_geometry* g) {
  return g && cr::check_geometry(g) == CR_OK ? cr::qsa_union_rows(g) : 0;
}

extern "C" cr_status cr_qsa_union_build(const cr_geometry* g, const cr_qsa_args* a, const cr_qsa_union* u, void* stream) {
  using namespace cr;
  if (cr_status s = qsa_validate(g, a, 1, CR_MAX_PREFILL_ROWS, "cr_qsa_union_build")) return s;
  CR_REQUIRE(u && u->list && u->count, "cr_qsa_union_build: null list or count");
  CR_REQUIRE(((uintptr_t)u->list & 7) == 0, "cr_qsa_union_build: list must be 8-byte aligned");
  return qsa_union_build_launch(g, *a, reinterpret_cast<int2*>(u->list), u->count, (cudaStream_t)stream);
}

extern "C" cr_status cr_qsa_prefill_attend(const cr_geometry* g, const cr_qsa_prefill_args* args, int skip, cr_out_format fmt, void* stream) {
  using namespace cr;
  if (cr_status s = check_part(g, args, skip, fmt, "cr_qsa_prefill_attend")) return s;
  return attend(g, args, output_rows(g, args->input, skip, fmt), skip, fmt, (cudaStream_t)stream);
}

extern "C" cr_status cr_qsa_prefill(const cr_geometry* g, const cr_qsa_prefill_args* args, int skip, cr_out_format fmt, void* stream_) {
  using namespace cr;
  if (cr_status s = check_part(g, args, skip, fmt, "cr_qsa_prefill")) return s;
  cudaStream_t stream = (cudaStream_t)stream_;
  // cache rows + query prep for the whole part (rows below skip get cache work only)
  if (cr_status s = qsa_prep_launch(g, &args->input, 1, 0, reinterpret_cast<__half*>(args->q_hi), skip, stream, false, skip == 0)) return s;
  const cr_qsa_args q = output_rows(g, args->input, skip, fmt);
  if (cr_status s = qsa_select_launch(g, &q, 1, stream, skip == 0)) return s;
  return attend(g, args, q, skip, fmt, stream);
}

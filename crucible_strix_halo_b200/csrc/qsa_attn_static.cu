// cr_qsa_attn_static: the decode / verify attention of cr_qsa_attn for callers that cannot hand over scratch memory: a
// serving process that has already given every spare byte of HBM to KV caches, a plugin loaded into someone else's process
// without access to that process's allocator, or code running while a stream capture is open on another thread.  The
// attention kernel merges its streams on chip, so nothing stands behind the entry point but the same launch; the limit on
// rows x heads is part of its contract.
#include <climits>
#include "qsa.cuh"

extern "C" cr_status cr_qsa_attn_static(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, cr_out_format fmt,
                                        void* stream) {
  using namespace cr;
  if (cr_status s = qsa_validate(g, spans, n_spans, CR_MAX_STEP_ROWS, "cr_qsa_attn_static")) return s;
  CR_REQUIRE(fmt == CR_OUT_RAW_F32 || fmt == CR_OUT_RAW_BF16 || fmt == CR_OUT_EXL3_WHT, "cr_qsa_attn_static: bad output format");
  size_t rows = 0;
  for (int s = 0; s < n_spans; ++s) {
    CR_REQUIRE(spans[s].out, "cr_qsa_attn_static: span %d has no output buffer", s);
    CR_REQUIRE(fmt != CR_OUT_EXL3_WHT || spans[s].suh_o, "cr_qsa_attn_static: span %d needs suh_o for the EXL3 output", s);
    CR_REQUIRE(fmt == CR_OUT_EXL3_WHT || spans[s].pack_rows == 0, "cr_qsa_attn_static: packed layout only with the EXL3 output");
    rows += (size_t)spans[s].R;
  }
  CR_REQUIRE(rows * (size_t)g->q_heads <= (size_t)CR_STATIC_ATTN_MAX_ROW_HEADS,
             "cr_qsa_attn_static: %zu rows x %d heads exceed the built-in scratch of %d (row, head) pairs; use cr_qsa_attn with caller scratch",
             rows, g->q_heads, CR_STATIC_ATTN_MAX_ROW_HEADS);
  return qsa_attn_launch(g, spans, n_spans, nullptr, 0, INT_MAX, fmt, (cudaStream_t)stream);
}

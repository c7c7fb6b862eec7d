// Snapshot / restore of a sequence's device state: the spans a host lists (fixed GDN state, conv rings, pending rows,
// compact raw rings, the open pool tile; or a whole conversation snapshot) are copied to or from one contiguous buffer
// in span order by ONE kernel per 1,200 spans, instead of one copy call per span
// (SlotCheckpointIO::Save / Restore, engine/runtime/slot_checkpoint_io.h:49-73; CopySnapshotSpans,
// engine/runtime/snapshot_bytes.h:692-704).  The copy is a grid-stride walk over 16 KB pieces of all spans together, so
// 133 spans of a 48-layer model between 2 KB and 2 MiB fill every SM evenly; each thread issues its four 128-bit
// loads before the first store.  HBM-bound: bytes read + bytes written = 2 x the spans' bytes.  The 132 spans (104 MB) of a
// 48-layer stream out and back: 86 us as two launches of at most 96 spans each way, 72 us as one (0.88 of the copy bandwidth).
#include "common.cuh"

namespace cr {

// Spans per launch: the table travels as a kernel parameter (24 bytes a span; the limit is 32,764 bytes).  A list of up to
// 96 spans takes the small table, which costs the launch less.
constexpr int kFewSpans = 96, kManySpans = 1200;
constexpr int kLoads = 4;                      // 128-bit loads a thread issues before its first store
constexpr int kPieceBytes = 256 * kLoads * 16;

template <int N>
struct CopyTable {
  const char* src[N];
  char* dst[N];
  unsigned first[N + 1];                       // first piece of span i; first[n] = pieces in all
  unsigned bytes16[N];                         // span length in 16-byte units
  int n;
};

template <int N>
__global__ void __launch_bounds__(256) state_copy_kernel(const __grid_constant__ CopyTable<N> T) {
  __shared__ unsigned first_s[N + 1];
  pdl_release();
  for (int i = threadIdx.x; i <= T.n; i += 256) first_s[i] = T.first[i];
  __syncthreads();
  pdl_wait();                                  // the table is read while the launch before this one still runs
  const unsigned total = first_s[T.n];
  for (unsigned piece = blockIdx.x; piece < total; piece += gridDim.x) {
    int lo = 0, hi = T.n - 1;                  // the span that holds this piece: last i with first[i] <= piece
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (first_s[mid] <= piece) lo = mid; else hi = mid - 1;
    }
    const unsigned unit0 = (piece - first_s[lo]) * (kPieceBytes / 16), units = T.bytes16[lo];
    const uint4* s = reinterpret_cast<const uint4*>(T.src[lo]) + unit0;
    uint4* d = reinterpret_cast<uint4*>(T.dst[lo]) + unit0;
    uint4 v[kLoads];
#pragma unroll
    for (int k = 0; k < kLoads; ++k) {
      const unsigned u = threadIdx.x + 256 * k;
      if (unit0 + u < units) v[k] = __ldcs(s + u);
    }
#pragma unroll
    for (int k = 0; k < kLoads; ++k) {
      const unsigned u = threadIdx.x + 256 * k;
      if (unit0 + u < units) __stcs(d + u, v[k]);
    }
  }
}

// One launch over the spans from i0 on; advances i0 and the offset in the buffer.
template <int N>
static cr_status copy_table(const cr_span* spans, int n, int& i0, char* buffer, size_t& offset, bool save, cudaStream_t stream) {
  CopyTable<N> T;
  T.n = 0;
  unsigned pieces = 0;
  for (; i0 < n && T.n < N; ++i0) {
    const cr_span& sp = spans[i0];
    if (sp.bytes == 0) continue;
    char* flat = buffer + offset;
    T.src[T.n] = save ? static_cast<const char*>(sp.ptr) : flat;
    T.dst[T.n] = save ? flat : static_cast<char*>(sp.ptr);
    T.first[T.n] = pieces;
    T.bytes16[T.n] = (unsigned)(sp.bytes / 16);
    pieces += (unsigned)((sp.bytes + kPieceBytes - 1) / kPieceBytes);
    offset += sp.bytes;
    ++T.n;
  }
  if (T.n == 0) return CR_OK;
  T.first[T.n] = pieces;
  const unsigned most = (unsigned)sm_count() * 8;
  CR_CUDA(launch_pdl(state_copy_kernel<N>, dim3(pieces < most ? pieces : most), dim3(256), 0, stream, T));
  CR_LAUNCH_CHECK("state_copy_kernel");
  return CR_OK;
}

static cr_status copy_spans(const cr_span* spans, int n, char* buffer, size_t buffer_bytes, bool save, cudaStream_t stream,
                            const char* who) {
  CR_REQUIRE(n >= 0 && (n == 0 || spans), "%s: null span list", who);
  CR_REQUIRE(n == 0 || buffer, "%s: null buffer", who);
  CR_REQUIRE(((uintptr_t)buffer & 15) == 0, "%s: the buffer must be 16-byte aligned", who);
  size_t total = 0;
  for (int i = 0; i < n; ++i) {
    CR_REQUIRE(spans[i].ptr || spans[i].bytes == 0, "%s: span %d is null", who, i);
    CR_REQUIRE(((uintptr_t)spans[i].ptr & 15) == 0 && spans[i].bytes % 16 == 0, "%s: span %d is not a multiple of 16 bytes at a 16-byte boundary",
               who, i);
    CR_REQUIRE(spans[i].bytes / 16 <= 0xffffffffull, "%s: span %d is too long", who, i);
    total += spans[i].bytes;
  }
  CR_REQUIRE(total <= buffer_bytes, "%s: the spans hold %zu bytes, the buffer %zu", who, total, buffer_bytes);
  size_t offset = 0;
  for (int i0 = 0; i0 < n;) {
    if (cr_status s = n - i0 <= kFewSpans ? copy_table<kFewSpans>(spans, n, i0, buffer, offset, save, stream)
                                          : copy_table<kManySpans>(spans, n, i0, buffer, offset, save, stream)) return s;
  }
  return CR_OK;
}
}  // namespace cr

extern "C" size_t cr_spans_bytes(const cr_span* spans, int n) {
  size_t total = 0;
  for (int i = 0; spans && i < n; ++i) total += spans[i].bytes;
  return total;
}

extern "C" cr_status cr_state_save(const cr_span* spans, int n, void* buffer, size_t buffer_bytes, void* stream) {
  return cr::copy_spans(spans, n, static_cast<char*>(buffer), buffer_bytes, true, (cudaStream_t)stream, "cr_state_save");
}

extern "C" cr_status cr_state_restore(const cr_span* spans, int n, const void* buffer, size_t buffer_bytes, void* stream) {
  return cr::copy_spans(spans, n, const_cast<char*>(static_cast<const char*>(buffer)), buffer_bytes, false, (cudaStream_t)stream,
                        "cr_state_restore");
}

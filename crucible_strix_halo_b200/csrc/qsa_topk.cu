// Exact top-512 of a row of indexer scores for sm_100a (the job of LaunchQsaTop, engine/layers/qsa_long.h:111-380):
// the 512 best blocks in the total order (score descending, block id ascending), emitted in ascending block id.
//
// Method: group maxima, pivot, filter, histogram, mark, compact.  One CTA of T = 1,024, 512 or 256 threads per row (many rows take the
// smaller ones), or a cluster of eight of 1,024 (long rows of steps; its own pivot, below).
//   1. Scores are >= +0, so their fp32 bit patterns order like unsigned integers (key = pattern + 1; 0 = no element).
//      The row falls into 1,024 groups: a thread reads every T-th element, or four where the row lies at 16 bytes, and keeps the maxima of
//      its 1,024 / T groups.
//   2. The pivot is a lower bound of the 512th largest of the 1024 group maxima: they are counted in 2,048 bins of the key
//      range below the largest, and a suffix scan finds the bin that holds the 512th.  At least 512 elements are >= the
//      bin's lower edge (those maxima themselves), so every element that can be among the best 512, ties included, is; with
//      unrelated scores about 700 are.
//   3. A second pass gathers the elements >= the pivot into a shared-memory list (warp-aggregated appends); the form for few rows of 14,337 to
//      32,768 blocks holds its elements in registers and reads the row once.
//   4. The same histogram over the list, between its known bounds, finds the bin of the 512th key: everything above is
//      taken, and the few elements inside the bin are ranked against each other (key, then index).  A crowded bin is
//      divided again, down to single keys; of equal keys the lowest indices are taken.
//   5. The taken elements set their bit in a bitmap over the row, which is compacted in index order: a prefix sum over
//      word popcounts gives every thread its output offset.
//   Rows that fit the list (4,096 elements; 3,072 with 512 or 256 threads) skip 1-3: every element goes into it.
//   Bound: block barriers of a latency chain (the row itself is read at L2 speed).  As 31-step bisections with a
//   block-wide count per bit, a row of 2,300 blocks took 16 us, 7 now; 2,048 rows of 65,536 blocks 268 -> 203 us (long
//   rows are read four elements at a time), of 8,192 blocks 125 -> 68 us.
//   When more elements pass the pivot than the list holds (long runs of equal scores), the row takes the slow exact path: the
//   same bisection over the whole row, counting with plain reductions, then the values above the 512th best pattern
//   plus its first ties in index order from a second bitmap.
// The same routine serves a whole row, a rank's block range (candidates with their scores, for split-KV across
// devices, engine/layers/qsa_long.h:228-234) and the merge of gathered candidates.
#include <climits>
#include <cooperative_groups.h>
#include "qsa.cuh"
#include "splits.h"

namespace cg = cooperative_groups;

namespace cr {

constexpr int kSelThreads = 1024;
constexpr int kMaxSelectCount = 262144;   // elements of one selection: the tie bitmap of the slow path takes the place of list and histogram
constexpr int kSortCap = 4096;            // entries of the candidate list (32 KB)
constexpr int kClusterRow = 20480;        // rows of at least this many blocks may take a cluster
constexpr int kHeldFrom = 14336, kHeldRow = 32 * kSelThreads;   // rows of one CTA that stay in registers: more blocks than the first, at most the second
constexpr int kShortCap = 3072;           // of the list of 256 and 512 threads, which take rows of many
constexpr int kShortRow = 14336;          // up to this many blocks (above, 512 threads are the quicker ones)

// ---- element sources ---------------------------------------------------------------------------------------
// A source maps an element index i in [0, count) to (bit pattern, block id, valid).  Index order is block-id order.
struct RowSource {                         // scores[i], block id = id_base + i
  const float* scores;
  int id_base;
  __device__ __forceinline__ bool get(int i, unsigned& bits) const { bits = __float_as_uint(scores[i]); return true; }
  __device__ __forceinline__ int id(int i) const { return id_base + i; }
  // Four consecutive elements, where the row starts at a 16-byte boundary and its buffer goes on to the next one.
  bool quads;
  __device__ __forceinline__ uint4 get4(int q) const { return reinterpret_cast<const uint4*>(scores)[q]; }
};
struct GatheredSource {                    // candidates of several ranks: element i = rank i / 512, slot i % 512
  const float* scores;
  const int* ids;
  size_t rank_stride;                      // elements between the lists of consecutive ranks
  __device__ __forceinline__ size_t at(int i) const { return (size_t)(i >> 9) * rank_stride + (i & 511); }
  __device__ __forceinline__ bool get(int i, unsigned& bits) const {
    const size_t a = at(i);
    if (ids[a] < 0) { bits = 0u; return false; }
    bits = __float_as_uint(scores[a]);
    return true;
  }
  __device__ __forceinline__ int id(int i) const { return ids[at(i)]; }
  static constexpr bool quads = false;
  __device__ __forceinline__ uint4 get4(int) const { return make_uint4(0u, 0u, 0u, 0u); }
};
__device__ __forceinline__ RowSource row_source(const cr_qsa_args& a, int r, int b0) {
  const float* s = a.scores + (size_t)r * a.sstride + b0;
  return RowSource{s, b0, ((uintptr_t)s & 15) == 0 && a.sstride % 4 == 0 && b0 % 4 == 0};
}

// ---- block-wide helpers ------------------------------------------------------------------------------------
template <int T>
__device__ __forceinline__ unsigned block_sum_u32(unsigned v, unsigned* red) {   // red: 33 words
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    unsigned t = threadIdx.x < T / 32 ? red[threadIdx.x] : 0u;
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) t += __shfl_xor_sync(0xffffffffu, t, m);
    if (threadIdx.x == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}
// Largest of one value per thread; one barrier (red: 32 words, free again after the caller's next barrier).
template <int T>
__device__ __forceinline__ unsigned block_max_u32(unsigned v, unsigned* red) {
  const unsigned m = __reduce_max_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  return __reduce_max_sync(0xffffffffu, (threadIdx.x & 31) < T / 32 ? red[threadIdx.x & 31] : 0u);
}
// Exclusive prefix sum of one value per thread over the block; one barrier before red is written, one after.
__device__ __forceinline__ unsigned block_exclusive_scan(unsigned v, unsigned* red) {
  const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned inc = v;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const unsigned o = __shfl_up_sync(0xffffffffu, inc, s);
    if (l >= s) inc += o;
  }
  __syncthreads();
  if (l == 31) red[w] = inc;
  __syncthreads();
  return __reduce_add_sync(0xffffffffu, l < w ? red[l] : 0u) + inc - v;
}
// Shared memory of one CTA: candidate list (32 KB), bitmap over the row's elements (count bits), small arrays.
struct SelectSmem {
  uint2* cand;                 // cap (key, index) pairs; the slow path keeps its tie bitmap here instead
  int cap;
  unsigned* bitmap;            // ceil(count / 32) words
  unsigned* red;               // 33 words
  unsigned* counter;           // 1 word
  int* hist;                   // kBins counters, zero between uses
  int* found;                  // 3 words
  uint2* ties;                 // kRankCap entries, in the place of the histogram once that has done its work
};

constexpr int kBatch = 8;      // loads a thread issues before it uses any of them

// Calls f(i, key) for the elements i = t, t + T, ... < count of this thread, key = bit pattern + 1 (0: no element).
// Loads are issued kBatch at a time.  WARP_UNIFORM: f is also called with key 0 for indices past the end, so that all
// lanes of a warp make the same number of calls (f may use warp-collective operations).
template <int T, bool WARP_UNIFORM, typename Src, typename F>
__device__ __forceinline__ void for_each_key(const Src& src, int count, F&& f) {
  const int lane = threadIdx.x & 31;
  for (int i0 = threadIdx.x; i0 - lane < count; i0 += T * kBatch) {   // the same trip count for a whole warp
    unsigned key[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int i = i0 + k * T;
      unsigned bits = 0u;
      key[k] = (i < count && src.get(i, bits)) ? bits + 1u : 0u;
    }
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int i = i0 + k * T;
      if (WARP_UNIFORM ? (i - lane < count) : (i < count)) f(i, key[k]);
    }
  }
}

// The same four elements at a time (src.quads): f(i, keys) for the elements i .. i + 3, keys past the end 0.  All lanes of a
// warp make the same number of calls.
template <int T, typename Src, typename F>
__device__ __forceinline__ void for_each_quad(const Src& src, int count, F&& f) {
  const int lane = threadIdx.x & 31, quads = (count + 3) >> 2;
  constexpr int kDeep = T >= 1024 ? 2 : 4;
  for (int q0 = threadIdx.x; q0 - lane < quads; q0 += T * kDeep) {
    uint4 v[kDeep];
#pragma unroll
    for (int k = 0; k < kDeep; ++k) {
      const int q = q0 + k * T;
      v[k] = q < quads ? src.get4(q) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int k = 0; k < kDeep; ++k) {
      const int q = q0 + k * T, i = 4 * q;
      if (q - lane >= quads) break;                                 // warp uniform
      f(i, make_uint4(i < count ? v[k].x + 1u : 0u, i + 1 < count ? v[k].y + 1u : 0u, i + 2 < count ? v[k].z + 1u : 0u, i + 3 < count ? v[k].w + 1u : 0u));
    }
  }
}

// ---- threshold by histogram ----------------------------------------------------------------------------------
constexpr int kBins = 2048;
constexpr int kRankCap = 512;              // elements of the threshold bin that are ranked against each other

static_assert(kShortCap <= kSortCap && kShortCap * 8 + kBins * 4 >= kMaxSelectCount / 8, "the tie bitmap of the longest row ends where the selection's begins");
static_assert(kRankCap * 8 <= kBins * 4, "the ranked elements fit the histogram's place");
struct Threshold { int bin, above, in_bin; };   // the bin that holds the want-th largest; elements in higher bins; in it
// sm.hist filled and visible.  The bin of the want-th largest counted element; bin = -1 when fewer were counted.  Two
// barriers; the histogram is zero again afterwards (visible after the caller's next barrier).
template <int T>
__device__ __forceinline__ Threshold find_threshold(const SelectSmem& sm, int want) {
  constexpr int PER = kBins / T;
  const int t = threadIdx.x, l = t & 31, w = t >> 5, first = kBins - 1 - t * PER;   // this thread's bins, descending
  int c[PER], sum = 0;
#pragma unroll
  for (int i = 0; i < PER; ++i) { c[i] = sm.hist[first - i]; sm.hist[first - i] = 0; sum += c[i]; }
  int inc = sum;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, inc, s);
    if (l >= s) inc += o;
  }
  if (l == 31) sm.red[w] = (unsigned)inc;
  if (t == 0) sm.found[0] = -1;
  __syncthreads();
  int before = (int)__reduce_add_sync(0xffffffffu, l < w ? sm.red[l] : 0u) + inc - sum;   // elements in higher bins
  if (before < want && before + sum >= want) {
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      if (before < want && before + c[i] >= want) { sm.found[0] = first - i; sm.found[1] = before; sm.found[2] = c[i]; }
      before += c[i];
    }
  }
  __syncthreads();
  return Threshold{sm.found[0], sm.found[1], sm.found[2]};
}
// Bits by which keys in [lo, hi] are shifted to fall into kBins bins.
__device__ __forceinline__ int bin_shift(unsigned lo, unsigned hi) {
  const unsigned span = hi > lo ? hi - lo : 0u;
  return span < (unsigned)kBins ? 0 : 21 - __clz(span);
}

// A lower bound of the want-th largest of G keys per thread (0: none), such that at least `want` keys are >= it; 1 when
// there are fewer.  largest: the largest of all keys.  sm.hist zero on entry.
template <int T, int G>
__device__ __forceinline__ unsigned pivot_of(const unsigned (&mine)[G], unsigned largest, int want, const SelectSmem& sm) {
  unsigned shift = 14;                                             // the four octaves below the largest key
#pragma unroll 1
  for (int round = 0; round < 2; ++round, shift = 20) {            // then everything
    const unsigned width = (unsigned)kBins << shift, lo = largest >= width ? largest - width + 1u : 1u;
#pragma unroll
    for (int k = 0; k < G; ++k)
      if (mine[k] >= lo) atomicAdd(&sm.hist[(mine[k] - lo) >> shift], 1);
    __syncthreads();
    const Threshold th = find_threshold<T>(sm, want);
    __syncthreads();
    if (th.bin >= 0) return lo + ((unsigned)th.bin << shift);
  }
  return 1u;
}

// The list sm.cand[0, m) holds (key, index) pairs that include the `want` best elements of the row (want <= m <= sm.cap),
// keys in [lo, hi]: marks those in sm.bitmap.  sm.hist zero and the list visible on entry; ends with a barrier.
template <int T>
__device__ __forceinline__ void select_from_list(int m, int want, const SelectSmem& sm, unsigned lo, unsigned hi) {
  const int t = threadIdx.x;
  // The first division covers the four octaves below the largest key (or less, if the list does); should they hold too few,
  // the whole range.
  const int full = bin_shift(lo, hi);
  int need = want, shift = full < 14 ? full : 14;
  unsigned first = full <= 14 ? lo : hi - ((unsigned)kBins << 14) + 1u, last;   // keys of the threshold bin
  Threshold th;
  for (;;) {
    const unsigned width = (unsigned)kBins << shift;
    for (int i = t; i < m; i += T) {
      const unsigned key = sm.cand[i].x, d = key - first;
      if (key >= first && key != 0u && d < width) atomicAdd(&sm.hist[d >> shift], 1);
    }
    __syncthreads();
    th = find_threshold<T>(sm, need);
    if (th.bin < 0) {
      shift = full; first = lo;
      __syncthreads();
      continue;
    }
    need -= th.above;
    first += (unsigned)th.bin << shift;
    last = first + ((1u << shift) - 1u);
    if (need == th.in_bin || th.in_bin <= kRankCap || shift == 0) break;
    shift = shift > 11 ? shift - 11 : 0;
    __syncthreads();                                               // the histogram is zero again for everybody
  }
  const bool all = need == th.in_bin, ranked = !all && th.in_bin <= kRankCap;
  if (ranked) {
    if (t == 0) *sm.counter = 0u;
    __syncthreads();
    for (int i = t; i < m; i += T) {
      const uint2 c = sm.cand[i];
      if (c.x >= first && c.x <= last && c.x != 0u) sm.ties[atomicAdd(sm.counter, 1u)] = c;
    }
    __syncthreads();
  }
  for (int i = t; i < m; i += T) {
    const uint2 c = sm.cand[i];
    if (c.x < first || c.x == 0u) continue;
    bool take = c.x > last || all;
    if (!take) {                                                   // inside the bin: better keys, then lower indices first
      const uint2* list = ranked ? sm.ties : sm.cand;              // a bin too crowded to rank holds one key only
      const int n = ranked ? th.in_bin : m;
      int before = 0;
      for (int j = 0; j < n; ++j) { const uint2 o = list[j]; before += (o.x > c.x && o.x <= last) || (o.x == c.x && o.y < c.y); }
      take = before < need;
    }
    if (take) atomicOr(&sm.bitmap[c.y >> 5], 1u << (c.y & 31));
  }
  __syncthreads();
}

template <int T, typename Src>
__device__ __forceinline__ void select_slow(const Src& src, int count, int want, const SelectSmem& sm);

// Marks the `want` best elements of [0, count) in sm.bitmap (bit i = element i selected).  want <= valid elements.
// HELD > 0: up to 4 HELD elements of a thread stay in registers between the two passes over the row, all of them in flight at once.
template <int T, int HELD = 0, typename Src>
__device__ __forceinline__ void select_mark(const Src& src, int count, int want, const SelectSmem& sm) {
  const int t = threadIdx.x, l = t & 31;
  constexpr int G = 1024 / T;                                      // groups of a thread: 1024 in the block
  const int words = (count + 31) >> 5;
  for (int i = t; i < words; i += T) sm.bitmap[i] = 0u;
  for (int i = t; i < kBins; i += T) sm.hist[i] = 0;
  if (t == 0) *sm.counter = 0u;
  unsigned pivot = 1u, mine = 0u, largest = 0u;                    // pivot 1: every element passes
  const bool held = HELD > 0 && count <= 4 * HELD * T;
  uint4 row[HELD > 0 ? HELD : 1];
  // The elements of row[k]: i, i + step, i + 2 step, i + 3 step, with i = held_at(k); quads, or where the row has none four that T lie between.
  const int step = src.quads ? 1 : T;
  auto held_at = [&](int k) { return (src.quads ? 4 * t : t) + 4 * k * T; };
  // f(i, keys) for the fours of this thread, all lanes of a warp alike
  auto held_fours = [&](auto&& f) {
#pragma unroll
    for (int k = 0; k < HELD; ++k)
      if (4 * k * T < count) f(held_at(k), row[k]);                // uniform
  };
  if (held) {
    if (src.quads) {
#pragma unroll
      for (int k = 0; k < HELD; ++k) row[k] = held_at(k) < count ? src.get4(t + k * T) : make_uint4(0u, 0u, 0u, 0u);
    } else {
#pragma unroll
      for (int k = 0; k < HELD; ++k) {
        const int i = held_at(k);
        row[k] = make_uint4(0u, 0u, 0u, 0u);
        if (i < count) src.get(i, row[k].x);
        if (i + T < count) src.get(i + T, row[k].y);
        if (i + 2 * T < count) src.get(i + 2 * T, row[k].z);
        if (i + 3 * T < count) src.get(i + 3 * T, row[k].w);
      }
    }
#pragma unroll
    for (int k = 0; k < HELD; ++k) {
      const int i = held_at(k);
      row[k] = make_uint4(i < count ? row[k].x + 1u : 0u, i + step < count ? row[k].y + 1u : 0u, i + 2 * step < count ? row[k].z + 1u : 0u,
                          i + 3 * step < count ? row[k].w + 1u : 0u);
    }
  }
  if (count > sm.cap) {
    unsigned group[G];
#pragma unroll
    for (int k = 0; k < G; ++k) group[k] = 0u;
    if (held) {
      held_fours([&](int, const uint4& k) { group[0] = max(max(max(group[0], k.x), max(k.y, k.z)), k.w); });
    } else if (src.quads) {
      for_each_quad<T>(src, count, [&](int, const uint4& k) {
        group[0] = max(group[0], k.x); group[1 % G] = max(group[1 % G], k.y); group[2 % G] = max(group[2 % G], k.z); group[3 % G] = max(group[3 % G], k.w);
      });
    } else {
      for_each_key<T, false>(src, count, [&](int i, unsigned key) {
#pragma unroll
        for (int k = 0; k < G; ++k)
          if (G == 1 || ((i / T) & (G - 1)) == k) group[k] = max(group[k], key);
      });
    }
#pragma unroll
    for (int k = 0; k < G; ++k) mine = max(mine, group[k]);
    largest = block_max_u32<T>(mine, sm.red);
    pivot = pivot_of<T, G>(group, largest, want, sm);
  } else {
    __syncthreads();
  }
  // ---- the elements >= pivot, as (key, index) pairs
  auto append = [&](int i, unsigned key) {
    const bool pass = key >= pivot;
    const unsigned m = __ballot_sync(0xffffffffu, pass);
    if (m) {
      unsigned base = 0u;
      if (l == 0) base = atomicAdd(sm.counter, (unsigned)__popc(m));
      base = __shfl_sync(0xffffffffu, base, 0);
      const unsigned at = base + __popc(m & ((1u << l) - 1u));
      if (pass && at < (unsigned)sm.cap) sm.cand[at] = make_uint2(key, (unsigned)i);
    }
  };
  auto append4 = [&](int i, const uint4& k, int by) {
    const unsigned best = max(max(k.x, k.y), max(k.z, k.w));
    mine = max(mine, best);
    if (!__any_sync(0xffffffffu, best >= pivot)) return;           // most quads of a long row
    append(i, k.x); append(i + by, k.y); append(i + 2 * by, k.z); append(i + 3 * by, k.w);
  };
  if (held) {
    held_fours([&](int i, const uint4& k) { append4(i, k, step); });
  } else if (src.quads) {
    for_each_quad<T>(src, count, [&](int i, const uint4& k) { append4(i, k, 1); });
  } else {
    for_each_key<T, true>(src, count, [&](int i, unsigned key) {
      mine = max(mine, key);
      append(i, key);
    });
  }
  if (count > sm.cap) __syncthreads();
  else largest = block_max_u32<T>(mine, sm.red);
  const int m = (int)*sm.counter;
  if (m >= want && m <= sm.cap) { select_from_list<T>(m, want, sm, pivot, largest); return; }
  select_slow<T>(src, count, want, sm);
}

// The slow exact path over the whole row; sm.bitmap zero on entry.
template <int T, typename Src>
__device__ __forceinline__ void select_slow(const Src& src, int count, int want, const SelectSmem& sm) {
  const int t = threadIdx.x, l = t & 31;
  const int words = (count + 31) >> 5;
  // ---- slow exact path: limit = the largest key with at least `want` elements >= limit
  unsigned limit = 0u;
  for (int bit = 30; bit >= 0; --bit) {
    const unsigned trial = limit | (1u << bit);
    unsigned c = 0u;
    for_each_key<T, false>(src, count, [&](int, unsigned key) { c += key >= trial; });
    if (block_sum_u32<T>(c, sm.red) >= (unsigned)want) limit = trial;
  }
  unsigned* ties = reinterpret_cast<unsigned*>(sm.cand);           // bitmap of the elements equal to limit: at most 32 KB, over the list and, past a short one, the histogram
  unsigned above = 0u;
  for_each_key<T, true>(src, count, [&](int i, unsigned key) {        // a warp covers one bitmap word per call
    const unsigned gt = __ballot_sync(0xffffffffu, key > limit), eq = __ballot_sync(0xffffffffu, key == limit);
    if (l == 0 && (i >> 5) < words) { sm.bitmap[i >> 5] = gt; ties[i >> 5] = eq; above += __popc(gt); }
  });
  const unsigned n_above = block_sum_u32<T>(above, sm.red);
  const unsigned need = (unsigned)want - n_above;                  // ties to take, lowest indices first
  // every thread owns a run of consecutive words: ties before the run decide how many of its own it takes
  const int per = (words + T - 1) / T, w0 = t * per, w1 = min(w0 + per, words);
  unsigned mine = 0u;
  for (int w = w0; w < w1; ++w) mine += __popc(ties[w]);
  unsigned before = block_exclusive_scan(mine, sm.red);
  for (int w = w0; w < w1 && before < need; ++w) {
    unsigned e = ties[w];
    const unsigned c = __popc(e);
    if (before + c > need) {                                       // keep only the lowest (need - before) set bits
      unsigned keep = 0u;
      for (unsigned k = need - before; k > 0; --k) { const unsigned low = e & (0u - e); keep |= low; e ^= low; }
      e = keep;
    }
    sm.bitmap[w] |= e;
    before += c;
  }
  __syncthreads();
}

// Writes the marked elements in index order: out_ids (and out_scores) get `want` entries.
template <int T, typename Src>
__device__ __forceinline__ void select_emit(const Src& src, int count, const SelectSmem& sm, int* out_ids, float* out_scores) {
  const int t = threadIdx.x;
  const int words = (count + 31) >> 5;
  const int per = (words + T - 1) / T, w0 = t * per, w1 = min(w0 + per, words);
  unsigned mine = 0u;
  for (int w = w0; w < w1; ++w) mine += __popc(sm.bitmap[w]);
  unsigned at = block_exclusive_scan(mine, sm.red);
  for (int w = w0; w < w1; ++w) {
    unsigned m = sm.bitmap[w];
    while (m) {
      const int i = (w << 5) + __ffs(m) - 1;
      m &= m - 1;
      out_ids[at] = src.id(i);
      if (out_scores) { unsigned bits; src.get(i, bits); out_scores[at] = __uint_as_float(bits); }
      ++at;
    }
  }
}

__device__ __forceinline__ SelectSmem carve(unsigned char* raw, int max_count, int cap = kSortCap) {
  SelectSmem sm;
  sm.cand = reinterpret_cast<uint2*>(raw);
  sm.cap = cap;
  sm.hist = reinterpret_cast<int*>(raw + (size_t)cap * 8);
  sm.ties = reinterpret_cast<uint2*>(sm.hist);
  sm.bitmap = reinterpret_cast<unsigned*>(sm.hist + kBins);
  sm.red = sm.bitmap + ((max_count + 31) >> 5);
  sm.counter = sm.red + 33;
  sm.found = reinterpret_cast<int*>(sm.counter + 1);
  return sm;
}
static size_t select_smem_bytes(int max_count, int cap = kSortCap) { return (size_t)cap * 8 + ((size_t)((max_count + 31) / 32) + 37 + kBins) * 4; }

// grid (rows, spans): the selection of one row.  Few rows: 1,024 threads each, what counts is the time of one.  In many a row is a chain
// of some sixteen short phases between barriers, and rows side by side on an SM are what fills it: five or six CTAs of 256 threads
// (40 registers, a list of 3,072 entries) or, where the rows are long, three of 512, so that the rows in flight are still in L2 when
// they are read again.  2,048 rows (two CTAs of 1,024 | 512 | 256 threads, us): 2,500 blocks 48 | 36 | 28, 8,192 blocks 69 | 51 | 47,
// 15,500 94 | 77 | 79, 25,500 123 | 105 | 117, 65,536 198 | 189 | 234.
// HELD (up to 32,768 blocks, a row to an SM): a thread's share of the row is loaded once, all at once, and stays in registers; by quads, or
// singly where the row does not lie at 16 bytes (three pitches in four): 15 rows of 20,479 blocks 10.8 and 11.2 us, 12.4 while the
// latter were read twice.
template <int T, int HELD = 0>
__global__ void __launch_bounds__(T, HELD > 0 ? 1 : T == 1024 ? 2 : T == 512 ? 3 : 6) qsa_topk_kernel(const __grid_constant__ QsaParams P, int max_count) {
  extern __shared__ __align__(16) unsigned char raw[];
  pdl_release();
  const cr_qsa_args& a = P.span[blockIdx.y];
  touch_params(a);
  pdl_wait();
  const int r = blockIdx.x;
  if (r >= a.R) return;
  const int nb = (a.pos0 + r + 1) / 4;
  if (nb <= CR_SEL_BLOCKS) { if (threadIdx.x == 0) a.nsel[r] = -1; return; }
  const SelectSmem sm = carve(raw, max_count, T == 1024 ? kSortCap : kShortCap);
  const RowSource src = row_source(a, r, 0);
  select_mark<T, HELD>(src, nb, CR_SEL_BLOCKS, sm);
  select_emit<T>(src, nb, sm, a.sel + (size_t)r * CR_SEL_BLOCKS, nullptr);
  if (threadIdx.x == 0) a.nsel[r] = CR_SEL_BLOCKS;
}

// Sorts the 32 values of a warp (one per lane) so that lane 0 holds the largest: a bitonic network of shuffles.
__device__ __forceinline__ unsigned warp_sort_desc(unsigned v) {
  const int l = threadIdx.x & 31;
#pragma unroll
  for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      const unsigned o = __shfl_xor_sync(0xffffffffu, v, j);
      const bool down = (l & k) == 0, low_lane = (l & j) == 0;       // in a descending run the lower lane keeps the larger value
      v = (low_lane == down) ? (v > o ? v : o) : (v < o ? v : o);
    }
  }
  return v;
}
// Descending bitonic sort of 128 values in shared memory by one warp.
__device__ __forceinline__ void warp_sort128_desc(unsigned* a) {
  const int l = threadIdx.x & 31;
  for (int k = 2; k <= 128; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      __syncwarp();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int q = l + 32 * h, i = ((q & ~(j - 1)) << 1) | (q & (j - 1));
        const unsigned x = a[i], y = a[i + j];
        if ((x < y) == ((i & k) == 0)) { a[i] = y; a[i + j] = x; }
      }
    }
  __syncwarp();
}

// The selection of one row by a cluster of 8 CTAs, for launches of few rows (decode and verify steps), where the time
// of one row is what counts: every CTA keeps an eighth of the row in registers (one read of the row, spread over 8
// SMs).  Pivot: every warp sorts its threads' maxima and lists the best four, a CTA offers the 64th largest of its 128
// listed values (64 of its elements are >= it; usually it is the CTA's 64th largest element), the cluster takes the
// smallest offer of its CTAs (512 elements are >= it; about 600 of 65,536 unrelated scores are).  Every CTA lists
// its elements >= the pivot in its own shared memory; CTA 0 collects the lists through distributed shared memory and
// finishes as the single-CTA kernel does.  grid (8 x rows, spans).
template <int PT>
__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(kSelThreads, 1) qsa_topk_cluster_kernel(const __grid_constant__ QsaParams P, int max_count) {
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ unsigned offer_s, max_s, count_s;                     // read by the other CTAs of the cluster
  __shared__ unsigned top4[128];
  pdl_release();
  const cr_qsa_args& a = P.span[blockIdx.y];
  touch_params(a);
  pdl_wait();
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int r = blockIdx.x / 8, t = threadIdx.x, l = t & 31;
  if (r >= a.R) return;                                            // the same for the whole cluster
  const int nb = (a.pos0 + r + 1) / 4;
  if (nb <= CR_SEL_BLOCKS) { if (rank == 0 && t == 0) a.nsel[r] = -1; return; }
  const SelectSmem sm = carve(raw, max_count);
  const float* sc = a.scores + (size_t)r * a.sstride;
  // An eighth of the row to each, to within one element: a CTA that holds less than the others would offer less than its 64th
  // largest, or nothing, and a pivot of nothing sends the row to the slow path.  (As multiples of 1,024 elements the eighths left the last
  // CTA short at three lengths in ten: 57 us at 21,000 blocks and 125 at 57,500, 10 and
  // 11 now.)
  const int base = topk_share(nb, rank), end = topk_share(nb, rank + 1);
  unsigned u[PT];
  unsigned mine = 0u;
#pragma unroll
  for (int k = 0; k < PT; ++k) {
    const int i = base + k * kSelThreads + t;
    u[k] = (base + k * kSelThreads < end && i < end) ? __float_as_uint(sc[i]) + 1u : 0u;   // the first test is the same for the CTA
    mine = u[k] > mine ? u[k] : mine;
  }
  const int words = (nb + 31) >> 5;
  if (rank == 0) {
    for (int i = t; i < words; i += kSelThreads) sm.bitmap[i] = 0u;
    for (int i = t; i < kBins; i += kSelThreads) sm.hist[i] = 0;
  }
  if (t == 0) *sm.counter = 0u;
  const unsigned sorted = warp_sort_desc(mine);
  if (l < 4) top4[(t >> 5) * 4 + l] = sorted;
  __syncthreads();
  if (t < 32) {
    warp_sort128_desc(top4);
    if (t == 0) { offer_s = top4[63]; max_s = top4[0]; }
  }
  cluster.sync();
  if (t < 8) {                                                     // eight threads fetch the offers of the eight CTAs
    unsigned x = *cluster.map_shared_rank(&offer_s, t), y = *cluster.map_shared_rank(&max_s, t);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      const unsigned xo = __shfl_xor_sync(0xffu, x, o), yo = __shfl_xor_sync(0xffu, y, o);
      x = xo < x ? xo : x;
      y = yo > y ? yo : y;
    }
    if (t == 0) { sm.red[0] = x; sm.red[1] = y; }
  }
  __syncthreads();
  unsigned pivot = sm.red[0];
  const unsigned largest = sm.red[1];
  if (pivot == 0u) pivot = 1u;                                     // rows of fewer than 4,096 blocks: everything passes, and the list holds it
#pragma unroll
  for (int k = 0; k < PT; ++k) {
    const bool pass = u[k] >= pivot && u[k] != 0u;
    const unsigned m = __ballot_sync(0xffffffffu, pass);
    if (m) {
      unsigned at = 0u;
      if (l == 0) at = atomicAdd(sm.counter, (unsigned)__popc(m));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << l) - 1u));
      if (pass && at < (unsigned)kSortCap) sm.cand[at] = make_uint2(u[k], (unsigned)(base + k * kSelThreads + t));
    }
  }
  __syncthreads();
  if (t == 0) count_s = *sm.counter;
  cluster.sync();
  if (rank == 0) {
    int total = 0, first[9];
#pragma unroll
    for (int c = 0; c < 8; ++c) { first[c] = total; total += (int)*cluster.map_shared_rank(&count_s, c); }
    first[8] = total;
    if (total <= kSortCap) {
      for (int c = 1; c < 8; ++c) {
        const uint2* theirs = cluster.map_shared_rank(sm.cand, c);
        for (int i = t; i < first[c + 1] - first[c]; i += kSelThreads) sm.cand[first[c] + i] = theirs[i];
      }
    }
    __syncthreads();
    const RowSource src = row_source(a, r, 0);
    if (total >= CR_SEL_BLOCKS && total <= kSortCap) select_from_list<kSelThreads>(total, CR_SEL_BLOCKS, sm, pivot, largest);
    else select_slow<kSelThreads>(src, nb, CR_SEL_BLOCKS, sm);
    select_emit<kSelThreads>(src, nb, sm, a.sel + (size_t)r * CR_SEL_BLOCKS, nullptr);
    if (t == 0) a.nsel[r] = CR_SEL_BLOCKS;
  }
  cluster.sync();                                                  // the lists stay until CTA 0 has copied them
}

// A rank's candidates among blocks [b0, b1): its best 512 (score, id), ascending id, unused slots -1.
__global__ void __launch_bounds__(kSelThreads, 2) qsa_candidates_kernel(const __grid_constant__ QsaParams P, int b0, int b1, float* cand_scores,
                                                                     int* cand_ids, int max_count) {
  extern __shared__ __align__(16) unsigned char raw[];
  const cr_qsa_args& a = P.span[0];
  const int r = blockIdx.x, t = threadIdx.x;
  const int nb = (a.pos0 + r + 1) / 4;
  float* cs = cand_scores + (size_t)r * CR_SEL_BLOCKS;
  int* ci = cand_ids + (size_t)r * CR_SEL_BLOCKS;
  const int count = min(nb, b1) - b0;
  if (nb <= CR_SEL_BLOCKS || count <= CR_SEL_BLOCKS) {              // dense row, or the rank owns at most 512 blocks: all of them
    if (t < CR_SEL_BLOCKS) {
      const bool have = nb > CR_SEL_BLOCKS && t < count;
      cs[t] = have ? a.scores[(size_t)r * a.sstride + b0 + t] : -1.f;
      ci[t] = have ? b0 + t : -1;
    }
    return;
  }
  const SelectSmem sm = carve(raw, max_count);
  const RowSource src = row_source(a, r, b0);
  select_mark<kSelThreads>(src, count, CR_SEL_BLOCKS, sm);
  select_emit<kSelThreads>(src, count, sm, ci, cs);
}

// Global selection from the gathered candidates [ranks][rows][512] of all ranks (ranks own ascending block ranges).
__global__ void __launch_bounds__(kSelThreads) qsa_merge_candidates_kernel(const __grid_constant__ QsaParams P, int ranks, const float* cand_scores,
                                                                           const int* cand_ids, int max_count) {
  extern __shared__ __align__(16) unsigned char raw[];
  const cr_qsa_args& a = P.span[0];
  const int r = blockIdx.x;
  const int nb = (a.pos0 + r + 1) / 4;
  if (nb <= CR_SEL_BLOCKS) { if (threadIdx.x == 0) a.nsel[r] = -1; return; }
  const SelectSmem sm = carve(raw, max_count);
  const size_t off = (size_t)r * CR_SEL_BLOCKS;
  const GatheredSource src{cand_scores + off, cand_ids + off, (size_t)a.R * CR_SEL_BLOCKS};
  select_mark<kSelThreads>(src, ranks * CR_SEL_BLOCKS, CR_SEL_BLOCKS, sm);
  select_emit<kSelThreads>(src, ranks * CR_SEL_BLOCKS, sm, a.sel + off, nullptr);
  if (threadIdx.x == 0) a.nsel[r] = CR_SEL_BLOCKS;
}

static int g_topk_clusters[64];                          // per device: clusters of 8 CTAs that run at once
static cr_status select_configure() {
  static PerDeviceOnce configured;
  return once_per_device(configured, [] {
    const int most = (int)select_smem_bytes(kMaxSelectCount);
    CR_CUDA(cudaFuncSetAttribute(qsa_topk_kernel<kSelThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CR_CUDA(cudaFuncSetAttribute(qsa_topk_kernel<kSelThreads, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CR_CUDA(cudaFuncSetAttribute(qsa_topk_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)select_smem_bytes(kShortRow, kShortCap)));
    CR_CUDA(cudaFuncSetAttribute(qsa_topk_kernel<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)select_smem_bytes(kMaxSelectCount, kShortCap)));
    CR_CUDA(cudaFuncSetAttribute(qsa_topk_cluster_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CR_CUDA(cudaFuncSetAttribute(qsa_topk_cluster_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CR_CUDA(cudaFuncSetAttribute(qsa_candidates_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CR_CUDA(cudaFuncSetAttribute(qsa_merge_candidates_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    int dev = 0;
    CR_CUDA(cudaGetDevice(&dev));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(8 * 64); cfg.blockDim = dim3(kSelThreads); cfg.dynamicSmemBytes = select_smem_bytes(65536);
    CR_CUDA(cudaOccupancyMaxActiveClusters(&g_topk_clusters[dev & 63], qsa_topk_cluster_kernel<8>, &cfg));
    return CR_OK;
  });
}

cr_status qsa_topk_launch(const cr_geometry* g, const cr_qsa_args* spans, int n_spans, cudaStream_t stream, bool dense_marked) {
  use_stream(stream);
  if (cr_status st = select_configure()) return st;
  for (int s0 = 0; s0 < n_spans; s0 += kMaxSpans) {
    const int n = n_spans - s0 < kMaxSpans ? n_spans - s0 : kMaxSpans;
    QsaParams P;
    qsa_fill_params(P, g, spans + s0, n);
    const int Rmax = qsa_max_rows(spans + s0, n);
    int nb_max = 0;
    for (int s = 0; s < n; ++s) nb_max = max(nb_max, (spans[s0 + s].pos0 + spans[s0 + s].R) / 4);
    CR_REQUIRE(nb_max <= kMaxSelectCount, "qsa select: %d blocks exceed the selectable range of %d", nb_max, kMaxSelectCount);
    if (dense_marked && nb_max <= CR_SEL_BLOCKS) continue;          // no row of these spans selects
    // Long rows take 8 SMs each while all clusters run at once (fifteen or so: 10 to 11.7 us at 12,000 to 65,536 blocks, 12.6 to 15.2 at
    // 70,000 to 262,144, whatever the length; 16 rows took 18 to 21, 36 rows 28 to 31).  A CTA per row: 20 us at 65,536 blocks, 12 at 32,768 with
    // the row held in registers (14.1 read twice), 10.5 at 20,000, 10 at 16,384, and 9.4 against 8.8 at 12,288, so that shorter rows are read
    // twice.  Rows too long for the registers take up to two waves of clusters: as quick alone, and beside another kernel the few CTAs
    // of the other form wait for their second reading (16 sessions at 262,144 with the GDN step on a stream of its own: 146 us a step, 161
    // with a CTA per row).
    const long long rows = (long long)Rmax * n;
    int dev = 0;
    CR_CUDA(cudaGetDevice(&dev));
    const int fit = g_topk_clusters[dev & 63];
    if (nb_max >= kClusterRow && rows <= (nb_max > kHeldRow ? 2 * fit : fit)) {
      if (nb_max <= 65536) CR_CUDA(launch_pdl(qsa_topk_cluster_kernel<8>, dim3(8 * Rmax, n), dim3(kSelThreads), select_smem_bytes(nb_max), stream, P, nb_max));
      else CR_CUDA(launch_pdl(qsa_topk_cluster_kernel<32>, dim3(8 * Rmax, n), dim3(kSelThreads), select_smem_bytes(nb_max), stream, P, nb_max));
      CR_LAUNCH_CHECK("qsa_topk_cluster_kernel");
      continue;
    }
    if (rows <= sm_count() && nb_max > kHeldFrom && nb_max <= kHeldRow)
      CR_CUDA(launch_pdl(qsa_topk_kernel<kSelThreads, 8>, dim3(Rmax, n), dim3(kSelThreads), select_smem_bytes(nb_max), stream, P, nb_max));
    else if (rows <= 2 * sm_count())                 // all rows are on the chip at once
      CR_CUDA(launch_pdl(qsa_topk_kernel<kSelThreads>, dim3(Rmax, n), dim3(kSelThreads), select_smem_bytes(nb_max), stream, P, nb_max));
    else if (nb_max <= kShortRow)
      CR_CUDA(launch_pdl(qsa_topk_kernel<256>, dim3(Rmax, n), dim3(256), select_smem_bytes(nb_max, kShortCap), stream, P, nb_max));
    else
      CR_CUDA(launch_pdl(qsa_topk_kernel<512>, dim3(Rmax, n), dim3(512), select_smem_bytes(nb_max, kShortCap), stream, P, nb_max));
    CR_LAUNCH_CHECK("qsa_topk_kernel");
  }
  return CR_OK;
}

}  // namespace cr

extern "C" cr_status cr_qsa_shard_candidates(const cr_geometry* g, const cr_qsa_args* a, int b0, int b1, float* cand_scores,
                                             int* cand_ids, void* stream) {
  using namespace cr;
  CR_REQUIRE(a && b0 >= 0 && b1 >= b0, "cr_qsa_shard_candidates: bad block range");
  if (cr_status s = qsa_validate(g, a, 1, CR_MAX_PREFILL_ROWS, "cr_qsa_shard_candidates", (b1 < (a->pos0 + a->R) / 4 ? b1 : (a->pos0 + a->R) / 4) - b0)) return s;
  CR_REQUIRE(cand_scores && cand_ids && b0 >= 0 && b1 >= b0 && b1 - b0 <= kMaxSelectCount, "cr_qsa_shard_candidates: bad block range or null output");
  if (cr_status st = select_configure()) return st;
  QsaParams P;
  qsa_fill_params(P, g, a, 1);
  use_stream((cudaStream_t)stream);
  const int most = b1 - b0 > 1 ? b1 - b0 : 1;
  qsa_candidates_kernel<<<a->R, kSelThreads, select_smem_bytes(most), (cudaStream_t)stream>>>(P, b0, b1, cand_scores, cand_ids, most);
  CR_LAUNCH_CHECK("qsa_candidates_kernel");
  return CR_OK;
}

extern "C" cr_status cr_qsa_shard_select(const cr_geometry* g, const cr_qsa_args* a, int b0, int b1, float* cand_scores, int* cand_ids,
                                         void* stream) {
  using namespace cr;
  CR_REQUIRE(a && b0 >= 0 && b1 >= b0, "cr_qsa_shard_select: bad block range");
  if (cr_status s = qsa_validate(g, a, 1, CR_MAX_PREFILL_ROWS, "cr_qsa_shard_select", (b1 < (a->pos0 + a->R) / 4 ? b1 : (a->pos0 + a->R) / 4) - b0)) return s;
  CR_REQUIRE(cand_scores && cand_ids && b0 >= 0 && b1 >= b0 && b1 - b0 <= kMaxSelectCount, "cr_qsa_shard_select: bad block range or null output");
  if (cr_status s = qsa_score_launch(g, a, 1, (cudaStream_t)stream, b0, b1)) return s;
  return cr_qsa_shard_candidates(g, a, b0, b1, cand_scores, cand_ids, stream);
}

extern "C" cr_status cr_qsa_merge_candidates(const cr_geometry* g, const cr_qsa_args* a, int ranks, const float* cand_scores,
                                             const int* cand_ids, void* stream) {
  using namespace cr;
  if (cr_status s = qsa_validate(g, a, 1, CR_MAX_PREFILL_ROWS, "cr_qsa_merge_candidates", 0)) return s;
  CR_REQUIRE(cand_scores && cand_ids && ranks >= 1 && ranks <= 16, "cr_qsa_merge_candidates: need 1..16 ranks and candidate buffers");
  if (cr_status st = select_configure()) return st;
  QsaParams P;
  qsa_fill_params(P, g, a, 1);
  use_stream((cudaStream_t)stream);
  const int most = ranks * CR_SEL_BLOCKS;
  qsa_merge_candidates_kernel<<<a->R, kSelThreads, select_smem_bytes(most), (cudaStream_t)stream>>>(P, ranks, cand_scores, cand_ids, most);
  CR_LAUNCH_CHECK("qsa_merge_candidates_kernel");
  return CR_OK;
}

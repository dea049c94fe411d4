// Parallel rows and parallel columns: hash the pivot-normalised live pattern
// of every row (column), sort by (hash, index), then resolve each hash group
// with an exact proportionality check.
//
// Reference: rules/rule_parallel_rows.cu:132-888 and
// rules/rule_parallel_columns.cu:158-1129.  The hash is the reference's FNV-1a
// fold (sequential, or XOR-aggregated when nnz > 32 m) so that groups, and
// therefore every decision, coincide with the reference's.  The reference's
// signature pre-filter only removes rows that cannot share a full hash group
// (and its audit checks exactly that), so hashing every live row gives the
// same groups.
#include <climits>

#include "engine.cuh"
#include "folding.hpp"
#include "scan.cuh"
#include "sort.hpp"

namespace gpp {

namespace {

constexpr uint64_t kFnvOffset = 0xcbf29ce484222325ULL;
constexpr uint64_t kFnvPrime = 0x100000001b3ULL;
__host__ __device__ __forceinline__ uint64_t mix(uint64_t h, uint64_t x) { return (h ^ x) * kFnvPrime; }
__device__ __forceinline__ uint64_t dbits(double v) { return uint64_t(__double_as_longlong(v)); }

// Row hash of one row (any schedule: the result depends only on the row).
struct RowHashArgs {
  const offset_t* ptr;
  const int32_t* idx;
  const double* val;
  const uint8_t* keep_row;
  const uint8_t* keep_col;
  double tol;
  bool use_xor;
  uint64_t* out;
};

__device__ void row_hash_thread(const RowHashArgs& g, int i) {
  if (!g.keep_row[i]) { g.out[i] = uint64_t(i); return; }
  offset_t first = -1, len = 0;
  for (offset_t p = g.ptr[i]; p < g.ptr[i + 1]; ++p)
    if (!g.keep_col || g.keep_col[g.idx[p]]) { if (first < 0) first = p; ++len; }
  if (len == 0 || fabs(g.val[first]) <= g.tol) { g.out[i] = mix(kFnvOffset, uint64_t(i)); return; }
  const double pivot = g.val[first];
  uint64_t h = mix(kFnvOffset, uint64_t(len)), agg = 0;
  for (offset_t p = first; p < g.ptr[i + 1]; ++p) {
    if (g.keep_col && !g.keep_col[g.idx[p]]) continue;
    const uint64_t b = dbits(g.val[p] / pivot);
    if (g.use_xor) agg ^= mix(mix(kFnvOffset, uint64_t(g.idx[p])), b);
    else h = mix(mix(h, uint64_t(g.idx[p])), b);
  }
  g.out[i] = g.use_xor ? mix(h, agg) : h;
}

// Long rows (past kLongRow stored entries) under the ordered fold, eight to a
// block.  The fold visits a row's entries in stored order, two dependent 64-bit multiplications
// each (about 75 us for a 5,000-entry row), so eight lanes of one warp fold a
// row each and do nothing else; the other seven warps form the next stage of
// the rows' (column, bits of value / pivot) pairs in shared memory meanwhile,
// removed columns marked.  One row to a block left the 2,000 such rows of the
// 29.8M-nnz LP to take turns (943 us for all rows of that model).
constexpr int kHashRows = 8, kHashStage = 112;   // 28 loaders a row, four entries each
struct HashStage {
  int32_t col[kHashRows][kHashStage + 1];
  uint64_t bits[kHashRows][kHashStage + 1];
};
__device__ void row_hash_block(const RowHashArgs& g, const int32_t* rows, int count, HashStage* stage) {
  __shared__ offset_t from_shared[kHashRows], end_shared[kHashRows];
  __shared__ double pivot_shared[kHashRows];
  __shared__ int len_shared[kHashRows];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  {   // a warp per row: its live length and first live entry (the pivot)
    const int i = warp < count ? rows[warp] : -1;
    const bool keep = i >= 0 && g.keep_row[i];
    const offset_t a = keep ? g.ptr[i] : 0, e = keep ? g.ptr[i + 1] : 0;
    int len = int(e - a);
    offset_t first = a;
    if (g.keep_col) {
      len = 0;
      first = -1;
      for (int at = 0; e - a > at; at += 128) {
        bool live[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          live[k] = e - a > at + 32 * k + lane && g.keep_col[__ldcs(g.idx + a + at + 32 * k + lane)];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const unsigned mask = __ballot_sync(0xffffffffu, live[k]);
          if (first < 0 && mask) first = a + at + 32 * k + (__ffs(mask) - 1);
          len += __popc(mask);
        }
      }
    }
    const bool trivial = !keep || len == 0 || fabs(g.val[first]) <= g.tol;
    if (lane == 0) {
      from_shared[warp] = trivial ? e : first;
      end_shared[warp] = e;
      pivot_shared[warp] = trivial ? 1.0 : g.val[first];
      len_shared[warp] = len;
      if (i >= 0 && trivial) g.out[i] = keep ? mix(kFnvOffset, uint64_t(i)) : uint64_t(i);
    }
  }
  __syncthreads();
  int chunks = 0;
#pragma unroll
  for (int r = 0; r < kHashRows; ++r)
    chunks = max(chunks, int((int64_t(end_shared[r]) - from_shared[r] + kHashStage - 1) / kHashStage));
  const bool folds = threadIdx.x < kHashRows;
  const int row = folds ? int(threadIdx.x) : (int(threadIdx.x) - 32) / 28, slot = (int(threadIdx.x) - 32) % 28;
  const offset_t from = row >= 0 && row < kHashRows ? from_shared[row] : 0;
  const offset_t end = row >= 0 && row < kHashRows ? end_shared[row] : 0;
  const double pivot = pivot_shared[row >= 0 && row < kHashRows ? row : 0];
  uint64_t h = folds ? mix(kFnvOffset, uint64_t(len_shared[row])) : 0;
  for (int c = 0; c <= chunks; ++c) {
    if (warp > 0 && c < chunks) {
      const int64_t base = int64_t(from) + int64_t(c) * kHashStage + slot;
      int col[4];
      double v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        col[k] = base + 28 * k < end ? __ldcs(g.idx + base + 28 * k) : -1;
        v[k] = base + 28 * k < end ? __ldcs(g.val + base + 28 * k) : 0.0;
      }
      if (g.keep_col) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (col[k] >= 0 && !g.keep_col[col[k]]) col[k] = -1;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        stage[c & 1].col[row][slot + 28 * k] = col[k];
        stage[c & 1].bits[row][slot + 28 * k] = dbits(v[k] / pivot);
      }
    }
    if (folds && c > 0) {
      const HashStage& last = stage[(c - 1) & 1];
      const int n = int(min(int64_t(kHashStage), int64_t(end) - from - int64_t(c - 1) * kHashStage));
#pragma unroll 8
      for (int k = 0; k < n; ++k) {
        const int32_t j = last.col[row][k];
        const uint64_t b = last.bits[row][k];
        if (j >= 0) h = mix(mix(h, uint64_t(j)), b);
      }
    }
    __syncthreads();
  }
  if (folds && row < count && from < end) g.out[rows[row]] = h;
  __syncthreads();
}

// A warp's 32 medium rows under the ordered fold, one to a lane, eight stored
// entries of each per round.  Eight lanes load a row's eight (four rows at a time),
// divide by its pivot and stage the pairs in shared memory, where the row's lane
// folds them in stored order (an entry's fold is a serial chain of 64-bit multiplies,
// so one lane runs it; a form in which all eight lanes of a row ran it over shuffles
// took 904 us at the 29.8M-nnz LP, this one 805).  A first sweep under a column mask
// finds the live length and the first live entry (the pivot).  Rounds last as
// long as the longest row; rows that have ended are passed over in fours.
struct RowStage {
  int32_t col[32 * 9];   // rows padded to 9 entries: no bank conflicts either way
  uint64_t bits[32 * 9];
};
__device__ void row_hash_rows(const RowHashArgs& g, int i, RowStage& stage) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, sub = lane >> 3, gl = lane & 7;
  const bool keep = i >= 0 && g.keep_row[i];
  const offset_t a = keep ? g.ptr[i] : 0, e = keep ? g.ptr[i + 1] : 0;
  int len = int(e - a);
  offset_t first = a;
  if (g.keep_col) {
    len = 0;
    first = -1;
    for (int at = 0;; at += 8) {
      if (!__any_sync(kAll, e - a > at)) break;
      int col[8];
      unsigned mine = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const offset_t ra = __shfl_sync(kAll, a, 4 * k + sub), re = __shfl_sync(kAll, e, 4 * k + sub);
        col[k] = re - ra > at + gl ? __ldcs(g.idx + ra + at + gl) : -1;
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const unsigned live = __ballot_sync(kAll, col[k] >= 0 && g.keep_col[max(col[k], 0)]);
        if (lane >> 2 == k) mine = live >> (8 * (lane & 3)) & 0xffu;
      }
      if (first < 0 && mine) first = a + at + (__ffs(mine) - 1);
      len += __popc(mine);
    }
  }
  const bool trivial = !keep || len == 0 || fabs(g.val[first]) <= g.tol;
  const double pivot = trivial ? 1.0 : g.val[first];
  const offset_t from = trivial ? e : first;
  uint64_t h = mix(kFnvOffset, uint64_t(len));
  for (int at = 0;; at += 8) {
    const unsigned need = __ballot_sync(kAll, e - from > at);
    if (!need) break;
    int col[8];
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const offset_t rf = __shfl_sync(kAll, from, 4 * k + sub), re = __shfl_sync(kAll, e, 4 * k + sub);
      const bool in = re - rf > at + gl;
      col[k] = in ? __ldcs(g.idx + rf + at + gl) : -1;
      v[k] = in ? __ldcs(g.val + rf + at + gl) : 0.0;
    }
    if (g.keep_col) {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (col[k] >= 0 && !g.keep_col[col[k]]) col[k] = -1;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const double by = __shfl_sync(kAll, pivot, 4 * k + sub);
      if (need >> (4 * k) & 15u) {
        const int slot = (4 * k + sub) * 9 + gl;
        stage.col[slot] = col[k];
        stage.bits[slot] = dbits(v[k] / by);
      }
    }
    __syncwarp();
    if (need >> lane & 1u) {
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const int32_t c = stage.col[lane * 9 + t];
        const uint64_t b = stage.bits[lane * 9 + t];
        if (c >= 0) h = mix(mix(h, uint64_t(c)), b);
      }
    }
    __syncwarp();
  }
  if (i >= 0) {
    if (!keep) g.out[i] = uint64_t(i);
    else if (trivial) g.out[i] = mix(kFnvOffset, uint64_t(i));
    else g.out[i] = h;
  }
}

// The ordered fold of few medium rows: four to a warp, eight lanes each, which all
// run the row's fold over shuffles.  The form above keeps eight times fewer warps
// busy, and each round of its warps is longer.  So this form while the grid has a warp
// for every four rows: 1,000 rows of 300 entries take 49 us (62 under a column mask),
// 91 (134) in the form above, 1,000 rows of 1,000 entries 108 (155) against 240 (382);
// 100,000 rows of 64 entries, more than that, 54 (76) above and 91 (106) in fours.
__device__ void row_hash_four(const RowHashArgs& g, int i) {
  constexpr unsigned kAll = 0xffffffffu;
  const int gl = threadIdx.x & 7, shift = int(threadIdx.x & 24);
  const bool keep = i >= 0 && g.keep_row[i];
  const offset_t a = keep ? g.ptr[i] : 0, e = keep ? g.ptr[i + 1] : 0;
  int len = int(e - a);
  offset_t first = a;
  if (g.keep_col) {
    len = 0;
    first = -1;
    for (int at = 0; __any_sync(kAll, e - a > at); at += 8) {
      const bool live = e - a > at + gl && g.keep_col[__ldcs(g.idx + a + at + gl)];
      const unsigned bits = __ballot_sync(kAll, live) >> shift & 0xffu;
      if (first < 0 && bits) first = a + at + (__ffs(bits) - 1);
      len += __popc(bits);
    }
  }
  const bool trivial = !keep || len == 0 || fabs(g.val[first]) <= g.tol;
  const double pivot = trivial ? 1.0 : g.val[first];
  const offset_t from = trivial ? e : first;
  uint64_t h = mix(kFnvOffset, uint64_t(len));
  for (int at = 0; __any_sync(kAll, e - from > at); at += 8) {
    const bool in = e - from > at + gl;
    const int col = in ? __ldcs(g.idx + from + at + gl) : -1;
    const double v = in ? __ldcs(g.val + from + at + gl) : 0.0;
    const bool live = in && (!g.keep_col || g.keep_col[col]);
    const uint64_t bits = live ? dbits(v / pivot) : 0;
    const unsigned mask = __ballot_sync(kAll, live) >> shift & 0xffu;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int c = __shfl_sync(kAll, col, t, 8);
      const uint64_t b = __shfl_sync(kAll, bits, t, 8);
      if (mask >> t & 1u) h = mix(mix(h, uint64_t(c)), b);
    }
  }
  if (gl == 0 && i >= 0) g.out[i] = !keep ? uint64_t(i) : trivial ? mix(kFnvOffset, uint64_t(i)) : h;
}

// The XOR aggregate (dense matrices) takes a row's entries in any order, so there
// is no fold to wait for: every lane of a row's group, eight lanes to a medium row
// and a block to a long one, aggregates its own entries, four in flight.  One lane to a
// row, as in the forms above, 200 rows of 20,000 entries took 956 us, 40 here, and
// 1,000 rows of 300 entries 93 against 29.
template <int W>
__device__ __forceinline__ uint64_t group_xor(uint64_t v) {
#pragma unroll
  for (int off = W / 2; off; off >>= 1) v ^= __shfl_xor_sync(0xffffffffu, v, off, W);
  return v;
}
// What a lane finds in its share of the row's entries.
struct LiveShare {
  int len = 0, first = INT_MAX;   // live entries, the first one's position in the row
};
__device__ __forceinline__ LiveShare live_share(const RowHashArgs& g, offset_t a, int size, int lane, int width) {
  LiveShare s;
  for (int64_t at = lane; at < size; at += 4 * width) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int64_t q = at + k * width;
      if (q < size && g.keep_col[__ldcs(g.idx + a + q)]) {
        ++s.len;
        s.first = min(s.first, int(q));
      }
    }
  }
  return s;
}
__device__ __forceinline__ uint64_t xor_share(const RowHashArgs& g, offset_t a, int size, double pivot, int lane,
                                              int width) {
  uint64_t agg = 0;
  for (int64_t at = lane; at < size; at += 4 * width) {
    int col[4];
    double v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int64_t q = at + k * width;
      col[k] = q < size ? __ldcs(g.idx + a + q) : -1;
      v[k] = q < size ? __ldcs(g.val + a + q) : 0.0;
    }
    if (g.keep_col) {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (col[k] >= 0 && !g.keep_col[col[k]]) col[k] = -1;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (col[k] >= 0) agg ^= mix(mix(kFnvOffset, uint64_t(col[k])), dbits(v[k] / pivot));
  }
  return agg;
}
__device__ __forceinline__ uint64_t xor_hash(const RowHashArgs& g, int i, bool keep, bool trivial, int len, uint64_t agg) {
  return !keep ? uint64_t(i) : trivial ? mix(kFnvOffset, uint64_t(i)) : mix(mix(kFnvOffset, uint64_t(len)), agg);
}
// Eight lanes a row; i < 0 for none.  All lanes of the warp call it.
__device__ void row_xor_group(const RowHashArgs& g, int i) {
  const int gl = threadIdx.x & 7;
  const bool keep = i >= 0 && g.keep_row[i];
  const offset_t a = keep ? g.ptr[i] : 0;
  const int size = keep ? int(g.ptr[i + 1] - a) : 0;
  int len = size, first = 0;
  if (g.keep_col) {
    const LiveShare s = live_share(g, a, size, gl, 8);
    len = s.len;
    first = s.first;
#pragma unroll
    for (int off = 4; off; off >>= 1) {
      len += __shfl_xor_sync(0xffffffffu, len, off, 8);
      first = min(first, __shfl_xor_sync(0xffffffffu, first, off, 8));
    }
  }
  const bool trivial = !keep || len == 0 || fabs(g.val[a + first]) <= g.tol;
  const uint64_t agg = group_xor<8>(trivial ? 0 : xor_share(g, a, size, g.val[a + first], gl, 8));
  if (gl == 0 && i >= 0) g.out[i] = xor_hash(g, i, keep, trivial, len, agg);
}
__device__ void row_xor_block(const RowHashArgs& g, int i) {
  __shared__ int lens[kThreads / 32], firsts[kThreads / 32];
  __shared__ uint64_t aggs[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool keep = g.keep_row[i] != 0;
  const offset_t a = g.ptr[i];
  const int size = keep ? int(g.ptr[i + 1] - a) : 0;
  int len = size, first = 0;
  if (g.keep_col) {
    const LiveShare s = live_share(g, a, size, threadIdx.x, kThreads);
    len = __reduce_add_sync(0xffffffffu, s.len);
    first = __reduce_min_sync(0xffffffffu, s.first);
    if (lane == 0) {
      lens[warp] = len;
      firsts[warp] = first;
    }
    __syncthreads();
    len = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
      len += lens[w];
      first = min(first, firsts[w]);
    }
  }
  const bool trivial = !keep || len == 0 || fabs(g.val[a + first]) <= g.tol;
  uint64_t agg = group_xor<32>(trivial ? 0 : xor_share(g, a, size, g.val[a + first], threadIdx.x, kThreads));
  if (lane == 0) aggs[warp] = agg;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < kThreads / 32; ++w) agg ^= aggs[w];
    g.out[i] = xor_hash(g, i, keep, trivial, len, agg);
  }
  __syncthreads();   // the shares are reused by the block's next row
}

// Blocks for the long rows, which take longest, then for the medium and the
// short ones.
struct HashRoles {
  int long_blocks, medium_blocks, short_blocks;
  int grid() const { return long_blocks + medium_blocks + short_blocks; }
};
HashRoles hash_roles(int rows, offset_t nnz, bool use_xor) {
  const int64_t long_rows = int64_t(nnz) / kLongRow + 1;   // at most
  return HashRoles{int(use_xor ? std::min<int64_t>(kNumSMs * 4, long_rows)
                               : std::min<int64_t>(kNumSMs * 2, (long_rows + kHashRows - 1) / kHashRows)),
                   int(std::min<int64_t>(kNumSMs * 8, (int64_t(rows) + 31) / 32)),
                   grid_stride_blocks(rows, kThreads, 16)};
}

template <bool Xor>
__global__ void __launch_bounds__(kThreads)
row_hash_kernel(int rows, RowHashArgs g, const int32_t* __restrict__ medium, const int32_t* __restrict__ longq,
                const int32_t* __restrict__ counts, HashRoles roles) {
  after_previous_kernel();
  int b = blockIdx.x;
  if constexpr (Xor) {
    if (b < roles.long_blocks) {
      for (int q = b; q < counts[1]; q += roles.long_blocks) row_xor_block(g, longq[q]);
      return;
    }
    b -= roles.long_blocks;
    if (b < roles.medium_blocks) {   // four rows to a warp
      const int nwarps = roles.medium_blocks * (kThreads / 32);
      const int nmedium = counts[0];
      for (int q0 = (b * (kThreads / 32) + int(threadIdx.x >> 5)) * 4; q0 < nmedium; q0 += nwarps * 4) {
        const int q = q0 + int(threadIdx.x & 31) / 8;
        row_xor_group(g, q < nmedium ? medium[q] : -1);
      }
      return;
    }
  } else {
    __shared__ union {
      HashStage block[2];
      RowStage warp[kThreads / 32];
    } stage;
    if (b < roles.long_blocks) {
      const int count = counts[1];
      for (int q = b * kHashRows; q < count; q += roles.long_blocks * kHashRows)
        row_hash_block(g, longq + q, min(kHashRows, count - q), stage.block);
      return;
    }
    b -= roles.long_blocks;
    if (b < roles.medium_blocks) {   // 32 rows to a warp, or four while there are warps
      const int nwarps = roles.medium_blocks * (kThreads / 32);
      const int nmedium = counts[0];
      if (nmedium <= nwarps * 4) {
        const int q0 = (b * (kThreads / 32) + int(threadIdx.x >> 5)) * 4, q = q0 + int(threadIdx.x & 31) / 8;
        if (q0 < nmedium) row_hash_four(g, q < nmedium ? medium[q] : -1);
        return;
      }
      for (int q0 = (b * (kThreads / 32) + int(threadIdx.x >> 5)) * 32; q0 < nmedium; q0 += nwarps * 32) {
        const int q = q0 + int(threadIdx.x & 31);
        row_hash_rows(g, q < nmedium ? medium[q] : -1, stage.warp[threadIdx.x >> 5]);
      }
      return;
    }
  }
  b -= roles.medium_blocks;
  for (int i = b * int(blockDim.x) + int(threadIdx.x); i < rows; i += roles.short_blocks * int(blockDim.x))
    if (g.ptr[i + 1] - g.ptr[i] <= kShortRow) row_hash_thread(g, i);
}
void launch_row_hash(const DevCsr& A, const RowHashArgs& g, cudaStream_t s) {
  const RowSchedule& sch = stored_schedule(A);
  const HashRoles roles = hash_roles(A.rows, A.nnz, g.use_xor);
  const double bytes = 4.0 * (A.rows + 1) + 12.0 * A.nnz + A.rows + (g.keep_col ? A.cols : 0) + 8.0 * A.rows;
  if (g.use_xor)
    GPP_LAUNCH_BYTES(row_hash_kernel<true>, bytes, roles.grid(), kThreads, 0, s, A.rows, g, sch.medium.p,
                     sch.long_rows.p, sch.counts.p, roles);
  else
    GPP_LAUNCH_BYTES(row_hash_kernel<false>, bytes, roles.grid(), kThreads, 0, s, A.rows, g, sch.medium.p,
                     sch.long_rows.p, sch.counts.p, roles);
}

// Repeated-hash filter.  Only a hash that two or more live items share can
// form a group, so only those items need sorting.  Every live item takes two
// positions in a bitmap from its mixed hash (the SplitMix64 finaliser, so the
// positions are spread whatever the row hash's low bits look like), sets them
// in `seen`, and marks a position in `twice` when it finds it already set.
// An item is a candidate when both of its positions are marked.  Items with
// equal hashes have equal positions, so every group of two or more is kept
// whole; a hash held once is kept only if both of its positions collide with
// other items (with 32 bitmap positions per item, about 0.4% of them).  The
// dropped items are groups of one, which the group kernels pass over, and the
// kept ones stay in (hash, index) order, so the groups found, their order and
// every record are those of the unfiltered sort.
__device__ __forceinline__ uint64_t mix_hash(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}
__global__ void mark_hash_bits(int n, const uint8_t* __restrict__ keep, const uint64_t* __restrict__ hash,
                               uint32_t* __restrict__ seen, uint32_t* __restrict__ twice, uint64_t bit_mask) {
  after_previous_kernel();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (!keep[i]) continue;
    const uint64_t z = mix_hash(hash[i]);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint64_t b = (k ? z >> 32 : z) & bit_mask;
      const uint32_t bit = 1u << (b & 31u);
      if (atomicOr(seen + (b >> 5), bit) & bit) atomicOr(twice + (b >> 5), bit);
    }
  }
}
__device__ __forceinline__ bool hash_may_repeat(uint64_t hash, const uint32_t* twice, uint64_t bit_mask) {
  const uint64_t z = mix_hash(hash);
  const uint64_t b0 = z & bit_mask, b1 = (z >> 32) & bit_mask;
  return (twice[b0 >> 5] >> (b0 & 31u) & 1u) && (twice[b1 >> 5] >> (b1 & 31u) & 1u);
}

// --- parallel rows ------------------------------------------------------------
struct LiveCursor {
  offset_t p, e;
  __device__ LiveCursor(offset_t a, offset_t b, const int32_t* idx, const uint8_t* keep) : p(a), e(b) { skip(idx, keep); }
  __device__ void skip(const int32_t* idx, const uint8_t* keep) { while (keep && p < e && !keep[idx[p]]) ++p; }
};

// _parallel_row_ratio (rule_parallel_rows.cu:346-377): a_i = ratio * a_k entrywise.
__device__ bool row_ratio(int i, int k, const offset_t* ptr, const int32_t* idx, const double* val, double tol,
                          const uint8_t* keep_col, double* out) {
  LiveCursor L(ptr[i], ptr[i + 1], idx, keep_col), R(ptr[k], ptr[k + 1], idx, keep_col);
  if (L.p == L.e && R.p == R.e) { *out = 1.0; return true; }
  double ratio = 0.0;
  bool set = false;
  for (; L.p < L.e && R.p < R.e; ++L.p, ++R.p, L.skip(idx, keep_col), R.skip(idx, keep_col)) {
    if (idx[L.p] != idx[R.p]) return false;
    const double ai = val[L.p], ak = val[R.p];
    if (!set) {
      if (fabs(ak) <= tol) return false;
      ratio = ai / ak;
      set = true;
    }
    if (fabs(ai - ratio * ak) > tol) return false;
  }
  *out = ratio;
  return set && L.p == L.e && R.p == R.e;
}

__device__ __forceinline__ void scaled_interval(double lo, double hi, double r, double* sl, double* su) {
  const double a = lo * r, b = hi * r;
  if (r >= 0.0) { *sl = a; *su = b; } else { *sl = b; *su = a; }
}

// _kernel_parallel_row_groups (rule_parallel_rows.cu:415-521): one thread per
// hash group, representative and merge order exactly as the reference.
__global__ void row_groups_kernel(int count, const uint64_t* __restrict__ sh, const int32_t* __restrict__ sr,
                                  const uint8_t* __restrict__ keep_row, const uint8_t* __restrict__ keep_col,
                                  double* AL, double* AU, const offset_t* __restrict__ ptr,
                                  const int32_t* __restrict__ idx, const double* __restrict__ val, double coeff_tol,
                                  double interval_tol, uint8_t* __restrict__ del, int32_t* __restrict__ merge_to,
                                  int32_t* __restrict__ step_out, double* __restrict__ rec_vals, Report report) {
  after_previous_kernel();
  uint32_t infeasible = 0;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < count && !infeasible; s += gridDim.x * blockDim.x) {
    const uint64_t hs = sh[s];
    if (s > 0 && sh[s - 1] == hs) continue;
    int e = s;
    while (e + 1 < count && sh[e + 1] == hs) ++e;
    if (e <= s) continue;
    int seed = -1;
    bool seed_eq = false;
    for (int a = s; a <= e; ++a) {
      const int row = sr[a];
      if (!keep_row[row]) continue;
      const bool eq = isfinite(AL[row]) && isfinite(AU[row]) && fabs(AL[row] - AU[row]) <= interval_tol;
      if (seed < 0 || (eq && !seed_eq)) { seed = row; seed_eq = eq; }
    }
    if (seed < 0) continue;
    int rep = seed;
    double rsl = AL[seed], rsu = AU[seed];
    for (int a = s; a <= e; ++a) {
      const int row = sr[a];
      if (row == seed || !keep_row[row]) continue;
      double r;
      if (!row_ratio(seed, row, ptr, idx, val, coeff_tol, keep_col, &r)) continue;
      double sl, su;
      scaled_interval(AL[row], AU[row], r, &sl, &su);
      if (rsl <= sl + interval_tol && su <= rsu + interval_tol) { rep = row; rsl = sl; rsu = su; }
    }
    double rl = AL[rep], ru = AU[rep];
    bool found = false;
    int step = 0;
    for (int a = s; a <= e; ++a) {
      const int row = sr[a];
      if (row == rep || !keep_row[row]) continue;
      double r;
      if (!row_ratio(rep, row, ptr, idx, val, coeff_tol, keep_col, &r)) continue;
      found = true;
      double sl, su;
      scaled_interval(AL[row], AU[row], r, &sl, &su);
      if (fmax(rl, sl) > fmin(ru, su) + interval_tol) { infeasible = 1; break; }
      ++step;
      merge_to[row] = rep;
      step_out[row] = step;
      rec_vals[5 * int64_t(row) + 0] = r;
      rec_vals[5 * int64_t(row) + 1] = rl;
      rec_vals[5 * int64_t(row) + 2] = ru;
      rec_vals[5 * int64_t(row) + 3] = AL[row];
      rec_vals[5 * int64_t(row) + 4] = AU[row];
      rl = fmax(rl, sl);
      ru = fmin(ru, su);
      del[row] = 1;
    }
    if (found && !infeasible) { AL[rep] = rl; AU[rep] = ru; }
  }
  post_flags(report, infeasible);
}

__global__ void pack_parallel_records(int64_t count, const int32_t* __restrict__ ids, const int32_t* __restrict__ first,
                                      const double* __restrict__ rec_vals, int type, int32_t* __restrict__ types,
                                      int64_t* __restrict__ is, int64_t* __restrict__ vs, int32_t* __restrict__ idx,
                                      double* __restrict__ val) {
  after_previous_kernel();
  for (int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; k <= count; k += int64_t(gridDim.x) * blockDim.x) {
    is[k] = 2 * k;
    vs[k] = 5 * k;
    if (k == count) continue;
    const int d = ids[k];
    types[k] = type;
    idx[2 * k + 0] = type == 4 ? first[d] : d;   // ParallelRow: (kept, deleted); ParallelColumn: (deleted, kept)
    idx[2 * k + 1] = type == 4 ? d : first[d];
    for (int t = 0; t < 5; ++t) val[5 * k + t] = rec_vals[5 * int64_t(d) + t];
  }
}

// --- parallel columns ---------------------------------------------------------
// _kernel_parallel_column_hashes (rule_parallel_columns.cu:189-240).
__global__ void col_hash_kernel(int n, const uint8_t* __restrict__ keep_col, const uint8_t* __restrict__ keep_row,
                                const offset_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                                const double* __restrict__ val, double tol, uint64_t* __restrict__ out) {
  after_previous_kernel();
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    if (!keep_col[j]) { out[j] = uint64_t(j); continue; }
    int len = 0;
    double pivot = 0.0;
    bool set = false;
    for (offset_t p = ptr[j]; p < ptr[j + 1]; ++p)
      if (keep_row[idx[p]] && fabs(val[p]) > tol) { ++len; if (!set) { pivot = val[p]; set = true; } }
    if (!set || len == 0) { out[j] = mix(kFnvOffset, uint64_t(j)); continue; }
    uint64_t h = mix(kFnvOffset, uint64_t(len));
    for (offset_t p = ptr[j]; p < ptr[j + 1]; ++p)
      if (keep_row[idx[p]] && fabs(val[p]) > tol) h = mix(mix(h, uint64_t(idx[p])), dbits(val[p] / pivot));
    out[j] = h;
  }
}

__device__ __forceinline__ offset_t next_live_col_entry(offset_t p, offset_t e, const int32_t* idx, const double* val,
                                                        const uint8_t* keep_row, double zt) {
  while (p < e && !(keep_row[idx[p]] && fabs(val[p]) > zt)) ++p;
  return p;
}

// _parallel_column_ratio (rule_parallel_columns.cu:262-321): a_k = ratio * a_j
// with a per-entry relative tolerance.
__device__ bool col_ratio(int j, int k, const offset_t* ptr, const int32_t* idx, const double* val,
                          const uint8_t* keep_row, double zt, double coeff_tol, double* out) {
  offset_t pj = ptr[j], pk = ptr[k];
  const offset_t ej = ptr[j + 1], ek = ptr[k + 1];
  double ratio = 0.0;
  bool set = false;
  for (;;) {
    pj = next_live_col_entry(pj, ej, idx, val, keep_row, zt);
    pk = next_live_col_entry(pk, ek, idx, val, keep_row, zt);
    if (pj >= ej || pk >= ek) break;
    if (idx[pj] != idx[pk]) return false;
    const double aj = val[pj], ak = val[pk];
    if (!set) {
      if (fabs(aj) <= zt) return false;
      ratio = ak / aj;
      if (fabs(ratio) <= zt || !isfinite(ratio)) return false;
      set = true;
    }
    const double expected = ratio * aj;
    const double scale = fmax(fabs(ak), fabs(expected));
    if (!isfinite(expected) || fabs(ak - expected) > coeff_tol * scale) return false;
    ++pj;
    ++pk;
  }
  pj = next_live_col_entry(pj, ej, idx, val, keep_row, zt);
  pk = next_live_col_entry(pk, ek, idx, val, keep_row, zt);
  if (pj < ej || pk < ek || !set) return false;
  *out = ratio;
  return true;
}

__device__ __forceinline__ bool ratio_guarded(double r, double max_abs) {
  const double a = fabs(r);
  return isfinite(max_abs) && (max_abs < 1.0 || a > max_abs || a * max_abs < 1.0);
}

// _kernel_count_small_high_ratio_parallel_groups (rule_parallel_columns.cu:400-467).
__global__ void count_guard_groups(int count, const uint64_t* __restrict__ sh, const int32_t* __restrict__ sc,
                                   const uint8_t* __restrict__ keep_col, const uint8_t* __restrict__ keep_row,
                                   const double* __restrict__ c, const offset_t* __restrict__ ptr,
                                   const int32_t* __restrict__ idx, const double* __restrict__ val, double zt,
                                   double coeff_tol, double obj_tol, double max_abs, int max_size, int stop_after,
                                   int32_t* __restrict__ out) {
  after_previous_kernel();
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < count; s += gridDim.x * blockDim.x) {
    // Early exit once enough groups are counted: a plain (volatile) read, as
    // an atomic read of one address from every thread serialises them.
    if (*(volatile int32_t*)out >= stop_after) return;
    const uint64_t hs = sh[s];
    if (s > 0 && sh[s - 1] == hs) continue;
    int e = s;
    while (e + 1 < count && sh[e + 1] == hs) ++e;
    const int size = e - s + 1;
    if (size < 2 || size > max_size) continue;
    bool hit = false;
    for (int a = s; a < e && !hit; ++a) {
      const int j = sc[a];
      if (!keep_col[j]) continue;
      for (int b = a + 1; b <= e; ++b) {
        const int k = sc[b];
        if (!keep_col[k]) continue;
        double r;
        if (!col_ratio(j, k, ptr, idx, val, keep_row, zt, coeff_tol, &r)) continue;
        if (fabs(c[k] - r * c[j]) > obj_tol) continue;
        if (max_abs < 1.0 || fabs(r) > max_abs || fabs(r) * max_abs < 1.0) { hit = true; break; }
      }
    }
    if (hit) atomicAdd(out, 1);
  }
}

// _kernel_parallel_column_groups (rule_parallel_columns.cu:470-628): the pairs
// (j, k) of a hash group in order; a merge moves j's bounds, which the next
// pairs of j see.  Whether a pair is proportional, and its cost gap, depends
// on the matrix alone, so a warp tests 32 partners k of j at once and then
// takes the pairs that act one after the other; a group of up to kGroupThread
// columns is one thread's.  (2,400 equal singleton columns of the coupling row
// in the replicated LPs were 4.1 ms of one thread.)
struct ColumnGroups {
  const int32_t* sc;
  const uint8_t *keep_col, *keep_row;
  const double* c;
  double *l, *u;
  const offset_t* ptr;
  const int32_t* idx;
  const double* val;
  double zt, coeff_tol, obj_tol;
  uint8_t *del, *fixed;
  double* fval;
  int32_t* merge_to;
  double* rec_vals;
};
enum ColumnAction : int { kNoAction = 0, kMerge, kFixK, kFixJ, kUnboundedPair };

// What the pair (j, k) with ratio r does given j's bounds; `at` receives the
// value a column is fixed at.
__device__ __forceinline__ ColumnAction column_action(const ColumnGroups& g, double gap, double r, double tl, double tu,
                                                      double sl, double su, double& at) {
  if (fabs(gap) <= g.obj_tol) return kMerge;
  bool k_lo = false, k_hi = false, j_lo = false, j_hi = false;
  if (gap > g.obj_tol) {
    if (r > 0.0) { k_lo = !isfinite(tu); j_hi = !isfinite(sl); }
    else { k_lo = !isfinite(tl); j_lo = !isfinite(sl); }
  } else {
    if (r > 0.0) { k_hi = !isfinite(tl); j_lo = !isfinite(su); }
    else { k_hi = !isfinite(tu); j_hi = !isfinite(su); }
  }
  if (k_lo || k_hi) {
    at = k_lo ? sl : su;
    return isfinite(at) ? kFixK : kUnboundedPair;
  }
  if (j_lo || j_hi) {
    at = j_lo ? tl : tu;
    return isfinite(at) ? kFixJ : kUnboundedPair;
  }
  return kNoAction;
}
// Carries the action out; for a merge j's bounds (tl, tu) move.
__device__ __forceinline__ void column_apply(const ColumnGroups& g, ColumnAction what, int j, int k, double r,
                                             double& tl, double& tu, double sl, double su, double at) {
  if (what == kMerge) {
    g.merge_to[k] = j;
    double* rec = g.rec_vals + 5 * int64_t(k);
    rec[0] = r; rec[1] = sl; rec[2] = su; rec[3] = tl; rec[4] = tu;
    double nl = -INFINITY, nu = INFINITY;
    if (r > 0.0) { if (isfinite(tl) && isfinite(sl)) nl = tl + r * sl; }
    else if (isfinite(tl) && isfinite(su)) nl = tl + r * su;
    if (r > 0.0) { if (isfinite(tu) && isfinite(su)) nu = tu + r * su; }
    else if (isfinite(tu) && isfinite(sl)) nu = tu + r * sl;
    tl = nl;
    tu = nu;
    g.l[j] = nl;
    g.u[j] = nu;
    g.del[k] = 1;
  } else if (what == kFixK) {
    g.fixed[k] = 1;
    g.fval[k] = at;
  } else if (what == kFixJ) {
    g.fixed[j] = 1;
    g.fval[j] = at;
  }
}
__device__ __forceinline__ uint32_t action_flag(ColumnAction what) {   // 1 unbounded, 2 merged, 4 fixed
  return what == kUnboundedPair ? 1u : what == kMerge ? 2u : what == kNoAction ? 0u : 4u;
}

constexpr int kGroupThread = 8;
__global__ void __launch_bounds__(kThreads)
col_groups_kernel(int count, const uint64_t* __restrict__ sh, ColumnGroups g, double max_abs,
                  const int32_t* __restrict__ guard, int guard_min, Report report) {
  after_previous_kernel();
  uint32_t found = 0;
  const int lane = threadIdx.x & 31;
  const double active_max = guard && *guard < guard_min ? INFINITY : max_abs;
  const int stride = gridDim.x * blockDim.x;
  const int64_t top = (int64_t(count) + stride - 1) / stride * stride;
  for (int64_t s64 = blockIdx.x * blockDim.x + threadIdx.x; s64 < top; s64 += stride) {
    const int s = int(s64);
    const bool head = s64 < count && (s == 0 || sh[s - 1] != sh[s]);
    int e = s;
    if (head)
      while (e + 1 < count && e - s < kGroupThread && sh[e + 1] == sh[s]) ++e;
    const bool large = head && e - s == kGroupThread;   // more than kGroupThread columns
    if (head && !large && e > s) {
      for (int a = s; a < e && !(found & 1u); ++a) {
        const int j = g.sc[a];
        if (!g.keep_col[j] || g.del[j] || g.fixed[j]) continue;
        double tl = g.l[j], tu = g.u[j];
        for (int b = a + 1; b <= e; ++b) {
          const int k = g.sc[b];
          if (!g.keep_col[k] || g.del[k] || g.fixed[k]) continue;
          double r, at = 0.0;
          if (!col_ratio(j, k, g.ptr, g.idx, g.val, g.keep_row, g.zt, g.coeff_tol, &r)) continue;
          if (ratio_guarded(r, active_max)) continue;
          const double sl = g.l[k], su = g.u[k];
          const ColumnAction what = column_action(g, g.c[k] - r * g.c[j], r, tl, tu, sl, su, at);
          found |= action_flag(what);
          if (what == kUnboundedPair) break;
          column_apply(g, what, j, k, r, tl, tu, sl, su, at);
          if (what == kFixJ) break;
        }
      }
    }
    unsigned rest = __ballot_sync(0xffffffffu, large);
    while (rest) {
      const int src = __ffs(rest) - 1;
      rest &= rest - 1;
      const int gs = __shfl_sync(0xffffffffu, s, src);
      const uint64_t hash = sh[gs];
      int ge = gs;   // last column of the group
      for (;;) {
        const int at = ge + 1 + lane;
        const unsigned same = __ballot_sync(0xffffffffu, at < count && sh[at] == hash);
        const int run = __ffs(~same) - 1;   // lanes from the first on
        ge += run < 0 ? 32 : run;
        if (run >= 0) break;
      }
      bool stop = false;
      for (int a = gs; a < ge && !stop; ++a) {
        const int j = g.sc[a];
        __syncwarp();
        if (!g.keep_col[j] || *(volatile uint8_t*)(g.del + j) || *(volatile uint8_t*)(g.fixed + j)) continue;
        double tl = g.l[j], tu = g.u[j];
        const double cj = g.c[j];
        bool done = false;   // j is fixed
        for (int first = a + 1; first <= ge && !done && !stop; first += 32) {
          const int b = first + lane;
          int k = -1;
          double r = 0.0, gap = 0.0, sl = 0.0, su = 0.0;
          bool pending = false;
          if (b <= ge) {
            k = g.sc[b];
            pending = g.keep_col[k] && !*(volatile uint8_t*)(g.del + k) && !*(volatile uint8_t*)(g.fixed + k) &&
                      col_ratio(j, k, g.ptr, g.idx, g.val, g.keep_row, g.zt, g.coeff_tol, &r) &&
                      !ratio_guarded(r, active_max);
            if (pending) {
              gap = g.c[k] - r * cj;
              sl = g.l[k];
              su = g.u[k];
            }
          }
          for (;;) {
            double at = 0.0;
            const ColumnAction what = pending ? column_action(g, gap, r, tl, tu, sl, su, at) : kNoAction;
            const unsigned acting = __ballot_sync(0xffffffffu, what != kNoAction);
            if (!acting) break;
            const int who = __ffs(acting) - 1;
            const ColumnAction act = ColumnAction(__shfl_sync(0xffffffffu, int(what), who));
            found |= action_flag(act);
            if (act == kUnboundedPair) { stop = true; break; }
            if (lane == who) column_apply(g, act, j, k, r, tl, tu, sl, su, at);
            tl = __shfl_sync(0xffffffffu, tl, who);
            tu = __shfl_sync(0xffffffffu, tu, who);
            if (act == kFixJ) { done = true; break; }
            if (lane <= who) pending = false;   // pairs up to this one are over
          }
        }
        __syncwarp();
      }
    }
  }
  post_flags(report, found);
}

__global__ void col_apply(int n, int m, const uint8_t* __restrict__ del, const uint8_t* __restrict__ fixed,
                          const double* __restrict__ fval, const double* __restrict__ c, const double* __restrict__ shift,
                          uint8_t* __restrict__ keep_col, double* __restrict__ l, double* __restrict__ u,
                          double* __restrict__ AL, double* __restrict__ AU, double* __restrict__ contrib) {
  after_previous_kernel();
  const int top = n > m ? n : m;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < top; q += gridDim.x * blockDim.x) {
    if (q < n) {
      contrib[q] = 0.0;
      if (del[q] || fixed[q]) {
        keep_col[q] = 0;
        if (fixed[q]) { l[q] = fval[q]; u[q] = fval[q]; contrib[q] = c[q] * fval[q]; }
      }
    }
    if (q < m && shift) { AL[q] -= shift[q]; AU[q] -= shift[q]; }
  }
}
// FixedVariable records: (col, kept rows), (value, c, coefficients).
__global__ void fixed_sizes(int n, const uint8_t* __restrict__ fx, const offset_t* __restrict__ at_ptr,
                            const int32_t* __restrict__ at_idx, const uint8_t* __restrict__ keep_row,
                            int64_t* __restrict__ recs, int64_t* __restrict__ nz) {
  after_previous_kernel();
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    int64_t c = 0;
    if (fx[j])
      for (offset_t p = at_ptr[j]; p < at_ptr[j + 1]; ++p) c += keep_row[at_idx[p]] != 0;
    recs[j] = fx[j] ? 1 : 0;
    nz[j] = c;
  }
}
__global__ void fixed_pack(int n, const uint8_t* __restrict__ fx, const offset_t* __restrict__ at_ptr,
                           const int32_t* __restrict__ at_idx, const double* __restrict__ at_val,
                           const uint8_t* __restrict__ keep_row, const double* __restrict__ fval,
                           const double* __restrict__ c, const int64_t* __restrict__ rpos,
                           const int64_t* __restrict__ npos, int32_t* __restrict__ types, int64_t* __restrict__ is,
                           int64_t* __restrict__ vs, int32_t* __restrict__ idx, double* __restrict__ val) {
  after_previous_kernel();
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    if (j == 0) { is[0] = 0; vs[0] = 0; }
    if (!fx[j]) continue;
    const int64_t k = rpos[j], base = npos[j];
    int64_t ip = k + base, vp = 2 * k + base;
    types[k] = 0;
    idx[ip++] = j;
    val[vp++] = fval[j];
    val[vp++] = c[j];
    for (offset_t p = at_ptr[j]; p < at_ptr[j + 1]; ++p)
      if (keep_row[at_idx[p]]) { idx[ip++] = at_idx[p]; val[vp++] = at_val[p]; }
    is[k + 1] = ip;
    vs[k + 1] = vp;
  }
}

// Sorted (hash, index) pairs of the live rows (columns) whose hash may be
// shared: all live items up to kRepeatFilterMin, past it the candidates of
// the repeated-hash filter.
constexpr int32_t kRepeatFilterMin = 32768;
int32_t sorted_live_hashes(const uint64_t* hash, const uint8_t* keep, int32_t n, DBuf<uint64_t>& keys,
                           DBuf<int32_t>& ids, cudaStream_t s) {
  // The pairs are packed by one selection into arrays for all items (their
  // number is known afterwards).
  keys.alloc(size_t(std::max(n, 1)), s);
  ids.alloc(size_t(std::max(n, 1)), s);
  const auto pack = [hash, out_keys = keys.p, out_ids = ids.p] __device__(int64_t i, int at, bool taken) {
    if (!taken) return;
    out_keys[at] = hash[i];
    out_ids[at] = int32_t(i);
  };
  int32_t count;
  if (n > kRepeatFilterMin) {
    // 32 bitmap positions per item, a power of two between 2^20 and 2^29.
    int lg = 20;
    while (lg < 29 && (int64_t(1) << lg) < 32 * int64_t(n)) ++lg;
    const size_t words = size_t(1) << (lg - 5);
    DBuf<uint32_t> bits(2 * words, s);
    bits.zero();
    const uint64_t bit_mask = (uint64_t(1) << lg) - 1;
    GPP_LAUNCH(mark_hash_bits, grid_stride_blocks(n), kThreads, 0, s, n, keep, hash, bits.p, bits.p + words,
               bit_mask);
    const uint32_t* twice = bits.p + words;
    count = select_and_count(
        n, [=] __device__(int64_t i) { return keep[i] && hash_may_repeat(hash[i], twice, bit_mask); }, pack, s);
  } else {
    count = select_and_count(n, [keep] __device__(int64_t i) { return keep[i] != 0; }, pack, s);
  }
  radix_sort_pairs(keys.p, ids.p, count, s);
  return count;
}

}  // namespace

void parallel_row_hashes(const DevCsr& A, const uint8_t* keep_row, const uint8_t* keep_col, int mode,
                         uint64_t* hashes, cudaStream_t s) {
  // compute_parallel_row_hashes (rule_parallel_rows.cu:583-627); mode < 0
  // picks XOR aggregation when nnz > 32 m.
  if (A.rows <= 0) return;
  const bool use_xor = mode >= 0 ? mode != 0 : int64_t(A.nnz) > 32LL * A.rows;
  DBuf<uint8_t> ones;
  if (!keep_row) {
    ones.alloc(size_t(A.rows), s);
    check(cudaMemsetAsync(ones.p, 1, size_t(A.rows), s), "keep all rows");
    keep_row = ones.p;
  }
  launch_row_hash(A, RowHashArgs{A.ptr, A.idx, A.val, keep_row, keep_col, 1e-10, use_xor, hashes}, s);
}

void rule_parallel_rows(Plan& plan, const WorkingLp& lp, const Stats&, const gpp_params& p) {
  // apply_rule_parallel_rows (rule_parallel_rows.cu:643-888).
  if (plan.has_infeasible || plan.has_unbounded) return;
  const int m = lp.m();
  if (m <= 1) return;
  auto s = ctx().stream;
  DBuf<uint64_t> hash(size_t(m), s);
  launch_row_hash(lp.A,
                  RowHashArgs{lp.A.ptr, lp.A.idx, lp.A.val, plan.keep_row.p, plan.keep_col.p, p.zero_tol,
                              int64_t(lp.A.nnz) > 32LL * m, hash.p},
                  s);
  DBuf<uint64_t> keys;
  DBuf<int32_t> ids;
  const int32_t count = sorted_live_hashes(hash.p, plan.keep_row.p, m, keys, ids, s);
  if (count <= 1) return;
  DBuf<uint8_t> del(size_t(m), s);
  DBuf<int32_t> merge_to(size_t(m), s), step(size_t(m), s);
  DBuf<double> rec(size_t(5) * size_t(m), s);
  del.zero();
  if (plan.save_committed) plan.save_committed();
  const Report report = ctx().open_report(1);
  GPP_LAUNCH(row_groups_kernel, grid_stride_blocks(count), kThreads, 0, s, count, keys.p, ids.p, plan.keep_row.p,
             plan.keep_col.p, plan.AL.p, plan.AU.p, lp.A.ptr, lp.A.idx, lp.A.val, p.zero_tol, p.feasibility_tol,
             del.p, merge_to.p, step.p, rec.p, report);
  if (ctx().await(report)[0]) { plan.has_infeasible = true; return; }
  DBuf<uint64_t> dkeys(size_t(m), s);
  DBuf<int32_t> dids(size_t(m), s);
  const int32_t deleted = select_and_count(
      m, [del = del.p] __device__(int64_t i) { return del[i] != 0; },
      [step = step.p, out_keys = dkeys.p, ids = dids.p, keep_row = plan.keep_row.p] __device__(int64_t i, int at,
                                                                                               bool taken) {
        if (!taken) return;
        out_keys[at] = (uint64_t(uint32_t(step[i])) << 32) | uint32_t(i);
        ids[at] = int32_t(i);
        keep_row[i] = 0;
      },
      s);
  if (!deleted) return;
  if (p.record_postsolve_tape) {
    // Records ordered by (merge step, deleted row) (rule_parallel_rows.cu:79-84).
    radix_sort_pairs(dkeys.p, dids.p, deleted, s, bits_up_to(deleted) << 32);   // rows already ascend
    PostsolveSegment seg = make_segment(deleted, 2 * int64_t(deleted), 5 * int64_t(deleted));
    GPP_LAUNCH(pack_parallel_records, grid_stride_blocks(deleted + 1), kThreads, 0, s, int64_t(deleted), dids.p,
               merge_to.p, rec.p, 4, seg.types.p, seg.is.p, seg.vs.p, seg.idx.p, seg.val.p);
    plan.tape.push_back(std::move(seg));
  }
  plan.has_row_action = plan.has_change = true;
}

void rule_parallel_columns(Plan& plan, const WorkingLp& lp, const Stats&, const gpp_params& p) {
  // apply_rule_parallel_columns (rule_parallel_columns.cu:725-1127).
  if (plan.has_infeasible || plan.has_unbounded) return;
  const int m = lp.m(), n = lp.n();
  if (n <= 1) return;
  auto s = ctx().stream;
  DBuf<uint64_t> hash(size_t(n), s);
  GPP_LAUNCH_BYTES(col_hash_kernel, 4.0 * (n + 1) + 12.0 * lp.AT.nnz + n + m + 8.0 * n, grid_stride_blocks(n),
                   kThreads, 0, s, n, plan.keep_col.p, plan.keep_row.p, lp.AT.ptr, lp.AT.idx, lp.AT.val, p.zero_tol,
                   hash.p);
  DBuf<uint64_t> keys;
  DBuf<int32_t> ids;
  const int32_t count = sorted_live_hashes(hash.p, plan.keep_col.p, n, keys, ids, s);
  if (count <= 1) return;
  const double coeff_tol = std::fmax(p.zero_tol, p.bound_tol), obj_tol = coeff_tol;
  const bool guard = std::isfinite(p.parallel_columns_max_abs_ratio) && p.parallel_columns_scale_guard_min_groups > 1;
  DBuf<int32_t> guard_groups;
  if (guard) {
    guard_groups.alloc(1, s);
    guard_groups.zero();
    GPP_LAUNCH(count_guard_groups, grid_stride_blocks(count), kThreads, 0, s, count, keys.p, ids.p, plan.keep_col.p,
               plan.keep_row.p, plan.c.p, lp.AT.ptr, lp.AT.idx, lp.AT.val, p.zero_tol, coeff_tol, obj_tol,
               p.parallel_columns_max_abs_ratio, p.parallel_columns_scale_guard_max_group_size,
               p.parallel_columns_scale_guard_min_groups, guard_groups.p);
  }
  DBuf<uint8_t> del(size_t(n), s), fixed(size_t(n), s);
  DBuf<double> fval(size_t(n), s), rec(size_t(5) * size_t(n), s), contrib(size_t(n), s);
  DBuf<int32_t> merge_to(size_t(n), s);
  del.zero();
  fixed.zero();
  if (plan.save_committed) plan.save_committed();
  const Report report = ctx().open_report(1);
  const ColumnGroups groups{ids.p,       plan.keep_col.p, plan.keep_row.p, plan.c.p, plan.l.p, plan.u.p, lp.AT.ptr,
                            lp.AT.idx,   lp.AT.val,       p.zero_tol,      coeff_tol, obj_tol,  del.p,    fixed.p,
                            fval.p,      merge_to.p,      rec.p};
  GPP_LAUNCH(col_groups_kernel, grid_stride_blocks(count), kThreads, 0, s, count, keys.p, groups,
             p.parallel_columns_max_abs_ratio, guard_groups.p, p.parallel_columns_scale_guard_min_groups, report);
  const uint32_t found = uint32_t(ctx().await(report)[0]);
  if (found & 1u) { plan.has_unbounded = true; return; }
  const bool merged = (found & 2u) != 0, any_fixed = (found & 4u) != 0;
  if (!merged && !any_fixed) return;
  if (merged && p.record_postsolve_tape) {
    // Records ordered by deleted column (rule_parallel_columns.cu:83-87).
    DBuf<int32_t> dids(size_t(n), s);
    const int32_t merges = select_and_count(
        n, [del = del.p] __device__(int64_t i) { return del[i] != 0; },
        [ids = dids.p] __device__(int64_t i, int at, bool taken) {
          if (taken) ids[at] = int32_t(i);
        },
        s);
    PostsolveSegment seg = make_segment(merges, 2 * int64_t(merges), 5 * int64_t(merges));
    GPP_LAUNCH(pack_parallel_records, grid_stride_blocks(merges + 1), kThreads, 0, s, int64_t(merges), dids.p,
               merge_to.p, rec.p, 3, seg.types.p, seg.is.p, seg.vs.p, seg.idx.p, seg.val.p);
    plan.tape.push_back(std::move(seg));
  }
  DBuf<double> shift;
  if (any_fixed) {
    if (p.record_postsolve_tape) {
      DBuf<int64_t> rc(size_t(n) + 1, s), nz(size_t(n) + 1, s), rpos(size_t(n) + 1, s), npos(size_t(n) + 1, s);
      GPP_LAUNCH(fixed_sizes, grid_stride_blocks(n), kThreads, 0, s, n, fixed.p, lp.AT.ptr, lp.AT.idx, plan.keep_row.p,
                 rc.p, nz.p);
      const auto [recs, nnz] = exclusive_scan_pair_i64(rc.p, rpos.p, nz.p, npos.p, n, s);
      PostsolveSegment seg = make_segment(recs, recs + nnz, 2 * recs + nnz);
      GPP_LAUNCH(fixed_pack, grid_stride_blocks(n), kThreads, 0, s, n, fixed.p, lp.AT.ptr, lp.AT.idx, lp.AT.val,
                 plan.keep_row.p, fval.p, plan.c.p, rpos.p, npos.p, seg.types.p, seg.is.p, seg.vs.p, seg.idx.p,
                 seg.val.p);
      plan.tape.push_back(std::move(seg));
    }
    shift.alloc(size_t(std::max(m, 1)), s);
    if (m) row_gather_shift(lp.A, lp.AT, plan.keep_row.p, fixed.p, fval.p, nullptr, shift.p, s);
    plan.has_row_action = true;
  }
  GPP_LAUNCH(col_apply, grid_stride_blocks(std::max(n, m)), kThreads, 0, s, n, m, del.p, fixed.p, fval.p, plan.c.p,
             any_fixed ? shift.p : nullptr, plan.keep_col.p, plan.l.p, plan.u.p, plan.AL.p, plan.AU.p, contrib.p);
  plan.obj_delta += any_fixed ? det_sum_later(contrib.p, nullptr, n, s) : LateValue{};
  plan.has_col_action = plan.has_change = true;
}

}  // namespace gpp

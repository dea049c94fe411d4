// Stream compaction / re-indexing of the working LP and the general transpose.
//
// Reference: apply_plan_to_working_lp / compact_csr_by_masks_gpu
// (cpp/src/presolve/gpu_presolve.cu:95-436,715-770,1793-1930) and
// transpose_csr64 (cpp/src/presolve/transpose64.cu:54-117).
//
// Materialisation compacts A and A^T with the same row/column maps.  A^T is
// kept row-sorted, and the old->new maps are monotone, so compacting A^T gives
// exactly cusparseCsr2cscEx2(compact(A)): the per-apply transpose becomes a
// second streaming pass.  The general transpose below is only needed for an
// input A^T that is not row-sorted and for matrices rebuilt by a rule.
#include "engine.cuh"
#include "scan.cuh"
#include "sort.hpp"

#include <algorithm>
#include <utility>

namespace gpp {

namespace {

// ---- entry-tiled compaction -------------------------------------------------
//
// The stored entries are cut into tiles of kCompactTile consecutive positions,
// one block per tile; each of its warps takes kCompactWarp of them, 32 at a
// time, so the index and value streams are read coalesced whatever the row
// lengths.  Rows come in through two bit arrays over the positions, set by one
// pass over the row pointers: where a row that holds entries starts, and
// whether it is kept; an entry's row is the last start at or before it, so a
// word of 32 positions needs a count of leading zeros per lane.  Ballots rank
// the kept entries, and as few entries go, a warp's kept entries leave as
// nearly contiguous stores straight from registers.  The copy is a stream
// compaction in stored order, so a kept entry's output position is the number
// of kept entries before it.  One pass does it: tiles are handed out in order
// by a ticket counter, each tile publishes its kept count as soon as it knows
// it, and looks back over its predecessors' published counts (a decoupled
// look-back) for its output offset.  The kept masks and offsets it leaves give
// every row its new pointer in a last pass over the rows, which also clears the
// bits again.  A and A^T of a materialisation are two sides of each launch.
//
// Bound by the rate of the one random access per entry, to the inner map (the
// 29.8M-nnz LP's columns and rows, about 250 us a side at 4 bytes of each 32
// fetched), then by the look-back; DRAM stays at a third of its rate.  Per tile
// three block barriers (the ticket, the warps' counts, the offset) against the
// ten of a form that ranked and staged over the block, which took 287 us.  A
// form whose warps walked the rows of their part stalled on long runs of empty
// rows (1.56 ms a launch on the QAP N = 30 relaxation, 0.06 ms now).
constexpr int kCompactRounds = 8;
constexpr int kCompactWarp = 32 * kCompactRounds;
constexpr int kCompactWarps = kThreads / 32;
constexpr int kCompactTile = kCompactWarp * kCompactWarps;

// One matrix to compact: rows by outer_map, entries by inner_map.
struct CompactSide {
  offset_t nnz;
  int rows, cols, tiles;
  const offset_t* ptr;
  const int32_t* idx;
  const double* val;
  const int32_t *outer_map, *inner_map;
  uint2* rows_at;       // per 32 positions: bits of the row starts (x) and of the kept ones (y)
  uint8_t* part_kept;   // per warp part: its first entry's row, where that row starts before it, is kept
  uint32_t* masks;      // per 32 positions: the kept entries
  int32_t* before;      // per warp part: the kept entries before it
  int32_t outer_new;
  offset_t* out_ptr;
  int32_t* out_idx;
  double* out_val;
};
struct CompactSides {
  CompactSide side[2];
};

// A row marks the parts that it reaches past its first one by its thread, or past
// kMarkThread parts by its warp: with a thread alone a row of 1 million entries took
// 132 us and one of 10 million 1,259 us, 6.2 and 11.0 so.
constexpr int kMarkThread = 32;
__global__ void compact_mark_rows(CompactSides sides) {
  after_previous_kernel();
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const CompactSide& s = sides.side[k];
    if (s.tiles == 0) continue;
    for (int64_t base = int64_t(blockIdx.x) * blockDim.x + threadIdx.x - lane; base < s.rows;
         base += int64_t(gridDim.x) * blockDim.x) {
      const int64_t r = base + lane;
      const int64_t a = r < s.rows ? s.ptr[r] : 0, e = r < s.rows ? s.ptr[r + 1] : 0;
      bool kept = false;
      int first = 0, last = 0;   // parts that begin inside the row
      if (a != e) {
        kept = s.outer_map[r] >= 0;
        const uint32_t bit = 1u << (a & 31);
        atomicOr(&s.rows_at[a >> 5].x, bit);
        if (kept) atomicOr(&s.rows_at[a >> 5].y, bit);
        first = int(a / kCompactWarp) + 1;
        last = int((e + kCompactWarp - 1) / kCompactWarp);
      }
      const bool wide = last - first > kMarkThread;
      if (!wide)
        for (int w = first; w < last; ++w) s.part_kept[w] = kept;
      for (unsigned rest = __ballot_sync(0xffffffffu, wide); rest; rest &= rest - 1) {
        const int src = __ffs(rest) - 1;
        const int f = __shfl_sync(0xffffffffu, first, src), l = __shfl_sync(0xffffffffu, last, src);
        const bool of_row = __shfl_sync(0xffffffffu, int(kept), src) != 0;
        for (int w = f + lane; w < l; w += 32) s.part_kept[w] = of_row;
      }
    }
  }
}

// New pointers of the kept rows (an empty row's is the kept entries before its
// position too), and the row bits cleared for the next compaction.
__global__ void compact_row_pointers(CompactSides sides) {
  after_previous_kernel();
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const CompactSide& s = sides.side[k];
    if (s.tiles == 0) continue;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < s.rows; r += gridDim.x * blockDim.x) {
      const int64_t a = s.ptr[r];
      if (a < s.nnz) s.rows_at[a >> 5] = make_uint2(0u, 0u);
      const int nr = s.outer_map[r];
      if (nr < 0) continue;
      if (a >= s.nnz) {   // past the last entry
        s.out_ptr[nr] = s.out_ptr[s.outer_new];
        continue;
      }
      const int64_t part = a / kCompactWarp;
      int kept = s.before[part];
      for (int64_t w = part * kCompactRounds; w < a >> 5; ++w) kept += __popc(s.masks[w]);
      kept += __popc(s.masks[a >> 5] & ((1u << (a & 31)) - 1u));
      s.out_ptr[nr] = kept;
    }
  }
}

// `words` (one per tile of both sides) and `counters` are zero at launch and
// again after it; the kept counts of both sides are posted to the host.
__global__ void __launch_bounds__(kThreads)
compact_tiles(CompactSides sides, unsigned long long* words, unsigned int* counters, int32_t* error, Report report) {
  after_previous_kernel();
  __shared__ int warp_counts[kCompactWarps];
  __shared__ long long tile_before;
  __shared__ unsigned int ticket;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int total_tiles = sides.side[0].tiles + sides.side[1].tiles;
  for (;;) {
    if (threadIdx.x == 0) ticket = atomicAdd(counters, 1u);
    __syncthreads();
    if (ticket >= unsigned(total_tiles)) break;   // block-uniform
    const bool second = int(ticket) >= sides.side[0].tiles;
    const CompactSide& s = sides.side[second ? 1 : 0];
    const int t = int(ticket) - (second ? sides.side[0].tiles : 0);
    const int64_t part = int64_t(t) * kCompactWarps + warp;
    const int64_t base = part * kCompactWarp;
    const int len = int(max(int64_t(0), min(int64_t(kCompactWarp), int64_t(s.nnz) - base)));
    int col[kCompactRounds];
    double v[kCompactRounds];
#pragma unroll
    for (int k = 0; k < kCompactRounds; ++k) col[k] = k * 32 + lane < len ? __ldcs(s.idx + base + k * 32 + lane) : -1;
#pragma unroll
    for (int k = 0; k < kCompactRounds; ++k) v[k] = k * 32 + lane < len ? __ldcs(s.val + base + k * 32 + lane) : 0.0;
    // The part's row bits, one word pair per lane of the first kCompactRounds.
    const bool has = lane < kCompactRounds && lane * 32 < len;
    const uint2 mine = has ? s.rows_at[base / 32 + lane] : make_uint2(0u, 0u);
    bool carry = len > 0 && s.part_kept[part];
#pragma unroll
    for (int k = 0; k < kCompactRounds; ++k) col[k] = col[k] >= 0 ? s.inner_map[col[k]] : -1;
    const unsigned up_to = 0xffffffffu >> (31 - lane);   // this lane and those before it
    int kept = 0;
    unsigned mask[kCompactRounds];
#pragma unroll
    for (int k = 0; k < kCompactRounds; ++k) {
      const unsigned starts = __shfl_sync(0xffffffffu, mine.x, k), keeps = __shfl_sync(0xffffffffu, mine.y, k);
      const unsigned at = starts & up_to;
      const bool row_kept = at ? (keeps >> (31 - __clz(at)) & 1u) != 0 : carry;
      if (starts) carry = (keeps >> (31 - __clz(starts)) & 1u) != 0;
      mask[k] = __ballot_sync(0xffffffffu, row_kept && col[k] >= 0);
      kept += __popc(mask[k]);
      if (lane == k) s.masks[base / 32 + k] = mask[k];
    }
    if (lane == 0) warp_counts[warp] = kept;
    __syncthreads();
    if (warp == 0) {
      int sum = 0;
#pragma unroll
      for (int w = 0; w < kCompactWarps; ++w) sum += warp_counts[w];
      const long long before =
          publish_and_look_back(words + (second ? sides.side[0].tiles : 0), t, s.tiles, sum, error);
      if (lane == 0) {
        tile_before = before;
        if (t == s.tiles - 1) {
          s.out_ptr[s.outer_new] = offset_t(before + sum);
          report.words[second ? 1 : 0] = int32_t(before + sum);
        }
      }
    }
    __syncthreads();
    int64_t out = tile_before;
#pragma unroll
    for (int w = 0; w < kCompactWarps; ++w) out += w < warp ? warp_counts[w] : 0;
    if (lane == 0) s.before[part] = int32_t(out);
#pragma unroll
    for (int k = 0; k < kCompactRounds; ++k) {
      if (mask[k] >> lane & 1u) {
        const int64_t o = out + __popc(mask[k] & ((1u << lane) - 1u));
        s.out_idx[o] = col[k];
        s.out_val[o] = v[k];
      }
      out += __popc(mask[k]);
    }
    __syncthreads();   // the counts and the ticket are reused by the next tile
  }
  leave_zeroed(words, total_tiles, counters);
  post_report(report);
}

__global__ void histogram(const int32_t* __restrict__ idx, offset_t nnz, int32_t* __restrict__ counts) {
  after_previous_kernel();
  for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < nnz; p += int64_t(gridDim.x) * blockDim.x)
    atomicAdd(counts + idx[p], 1);
}
// Longest column (the histogram's largest count), one atomic per warp.
__global__ void longest_count(const int32_t* __restrict__ counts, int n, int32_t* __restrict__ out) {
  after_previous_kernel();
  int32_t best = 0;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) best = max(best, counts[j]);
  best = __reduce_max_sync(0xffffffffu, best);
  if ((threadIdx.x & 31) == 0 && best > 0) atomicMax(out, best);
}
// Short-column transpose: each stored position goes to a slot of its column
// through an atomic cursor (slot order within a column is arbitrary), then
// every column's positions are put back in ascending order, which is the
// stored (row-major) order: the same result as the stable sort.
constexpr int kShortColumn = 64;
__global__ void place_positions(offset_t nnz, const int32_t* __restrict__ idx, int32_t* __restrict__ cursor,
                                int32_t* __restrict__ pos) {
  after_previous_kernel();
  for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < nnz; p += int64_t(gridDim.x) * blockDim.x)
    pos[atomicAdd(cursor + idx[p], 1)] = int32_t(p);
}
__global__ void order_columns(int n, const offset_t* __restrict__ ptr, int32_t* __restrict__ pos) {
  after_previous_kernel();
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const offset_t first = ptr[j];
    const int len = int(ptr[j + 1] - first);
    if (len < 2) continue;
    int32_t a[kShortColumn];
    for (int k = 0; k < len; ++k) a[k] = pos[first + k];
    for (int k = 1; k < len; ++k) {   // insertion sort: columns hold at most kShortColumn entries
      const int32_t v = a[k];
      int q = k - 1;
      while (q >= 0 && a[q] > v) { a[q + 1] = a[q]; --q; }
      a[q + 1] = v;
    }
    for (int k = 0; k < len; ++k) pos[first + k] = a[k];
  }
}
// Column keys and entry positions of M, in stored (row-major) order.
__global__ void transpose_keys(offset_t nnz, const int32_t* __restrict__ idx, uint64_t* __restrict__ keys,
                               int32_t* __restrict__ pos) {
  after_previous_kernel();
  for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < nnz; p += int64_t(gridDim.x) * blockDim.x) {
    keys[p] = uint64_t(uint32_t(idx[p]));
    pos[p] = int32_t(p);
  }
}
// Row of every stored entry: one warp per row writes its run.
__global__ void row_of_entry(int rows, const offset_t* __restrict__ ptr, int32_t* __restrict__ row) {
  after_previous_kernel();
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  for (int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += warps)
    for (offset_t p = ptr[r] + lane; p < ptr[r + 1]; p += 32) row[p] = r;
}
// Entries in (column, row) order: gather their rows and values.
__global__ void transpose_gather(offset_t nnz, const int32_t* __restrict__ pos, const int32_t* __restrict__ row,
                                 const double* __restrict__ val, int32_t* __restrict__ out_idx,
                                 double* __restrict__ out_val) {
  after_previous_kernel();
  for (int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; q < nnz; q += int64_t(gridDim.x) * blockDim.x) {
    const int32_t p = pos[q];
    out_idx[q] = row[p];
    out_val[q] = val[p];
  }
}

// Four rows per warp, eight lanes per row, each lane comparing the pairs
// (p - 1, p) of its stride.
__global__ void check_sorted(int rows, const offset_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                             int32_t* bad) {
  after_previous_kernel();
  const int g = threadIdx.x & 7;
  const int groups = gridDim.x * (blockDim.x >> 3);
  for (int r = blockIdx.x * (blockDim.x >> 3) + (threadIdx.x >> 3); r < rows; r += groups)
    for (offset_t p = ptr[r] + 1 + g; p < ptr[r + 1]; p += 8)
      if (idx[p - 1] >= idx[p]) { atomicExch(bad, 1); break; }
}

// Structure of an uploaded CSR: pointers start at 0, end at nnz and never
// decrease; every inner index lies in [0, cols).  Any violation sets *bad.
__global__ void check_csr_structure(int rows, int cols, offset_t nnz, const offset_t* __restrict__ ptr,
                                    const int32_t* __restrict__ idx, int32_t* bad) {
  after_previous_kernel();
  const int64_t top = int64_t(rows) + 1 > int64_t(nnz) ? int64_t(rows) + 1 : int64_t(nnz);
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < top; i += int64_t(gridDim.x) * blockDim.x) {
    bool fail = false;
    if (i <= rows) {
      const offset_t p = ptr[i];
      if (i == 0 ? p != 0 : p < ptr[i - 1]) fail = true;
      if (i == rows && p != nnz) fail = true;
    }
    if (i < nnz) {
      const int32_t c = idx[i];
      if (c < 0 || c >= cols) fail = true;
    }
    if (fail) atomicExch(bad, 1);
  }
}

}  // namespace

// Old -> new map of a mask, straight from its bytes: a kept item's rank, -1
// for a dropped one; returns the number kept.
int32_t build_old_to_new(const uint8_t* keep, int32_t n, int32_t* old_to_new, cudaStream_t s) {
  return select_and_count(
      n, [keep] __device__(int64_t i) { return keep[i] != 0; },
      [old_to_new] __device__(int64_t i, int at, bool kept) { old_to_new[i] = kept ? at : -1; }, s);
}

std::pair<int32_t, int32_t> build_old_to_new_pair(const uint8_t* keep_row, int32_t m, int32_t* row_map,
                                                  const uint8_t* keep_col, int32_t n, int32_t* col_map,
                                                  cudaStream_t s) {
  // Both masks in one launch, as the prefix sums of m + n items.
  auto& c = ctx();
  const uint32_t seq = c.open_mail();
  Mailbox* mail = c.box(seq);
  scan_items<int32_t, 2>(
      int64_t(m) + n,
      [=] __device__(int64_t i, int32_t(&v)[2]) {
        if (i < m) v[0] = keep_row[i] != 0;
        else v[1] = keep_col[i - m] != 0;
      },
      [=] __device__(int64_t i, const int32_t(&before)[2], const int32_t(&v)[2]) {
        if (i < m) row_map[i] = v[0] ? before[0] : -1;
        else col_map[i - m] = v[1] ? before[1] : -1;
      },
      [=] __device__(const int32_t(&sum)[2]) { post_values(mail, seq, sum[0], sum[1]); }, s);
  const int64_t* kept = c.await(mail, seq, "kept rows and columns");
  return {int32_t(kept[0]), int32_t(kept[1])};
}

namespace {
// The output of compacting M, its arrays sized for all stored entries (nothing
// waits for the kept count before the copy), and the side that fills it; an
// output without rows, columns or entries is only given its zero pointers.
DevCsr compact_output(const DevCsr& M, const int32_t* outer_map, int32_t outer_new, const int32_t* inner_map,
                      int32_t inner_new, CompactSide& side, cudaStream_t s) {
  DevCsr out;
  out.rows = outer_new;
  out.cols = inner_new;
  out.ptr = dalloc<offset_t>(size_t(outer_new) + 1);
  if (outer_new == 0 || inner_new == 0 || M.nnz == 0) {
    check(cudaMemsetAsync(out.ptr, 0, sizeof(offset_t) * (size_t(outer_new) + 1), s), "compact empty ptr");
    return out;
  }
  out.idx = dalloc<int32_t>(size_t(M.nnz));
  out.val = dalloc<double>(size_t(M.nnz));
  side.nnz = M.nnz;
  side.rows = M.rows;
  side.cols = M.cols;
  side.tiles = int((int64_t(M.nnz) + kCompactTile - 1) / kCompactTile);
  side.ptr = M.ptr;
  side.idx = M.idx;
  side.val = M.val;
  side.outer_map = outer_map;
  side.inner_map = inner_map;
  side.outer_new = outer_new;
  side.out_ptr = out.ptr;
  side.out_idx = out.idx;
  side.out_val = out.val;
  return out;
}

// Compacts the sides that hold entries; their kept counts go to `out`.
void compact_sides(CompactSides& sides, DevCsr* const (&out)[2], cudaStream_t s) {
  const int tiles = sides.side[0].tiles + sides.side[1].tiles;
  if (tiles == 0) return;
  const size_t parts = size_t(tiles) * kCompactWarps, words32 = parts * kCompactRounds;
  auto& c = ctx();
  // Row bits, zero before and after: up to 1 MB stays with the context (a memset
  // of a small model's costs as much as its kernels), past that they are the call's.
  constexpr size_t kKeptRowBits = size_t(1) << 17;
  DBuf<uint2> large_bits;
  uint2* row_bits;
  if (words32 > kKeptRowBits) {
    large_bits.alloc(words32, s);
    large_bits.zero();
    row_bits = large_bits.p;
  } else {
    if (c.row_bits_words < words32) {
      const size_t grown = std::min(kKeptRowBits, std::max(words32, 2 * c.row_bits_words));
      uint2* p = dalloc<uint2>(grown);
      dfree(std::exchange(c.row_bits, p));
      c.row_bits_words = grown;
      check(cudaMemsetAsync(p, 0, sizeof(uint2) * grown, s), "row bits");
    }
    row_bits = c.row_bits;
  }
  DBuf<uint32_t> masks(words32, s);
  DBuf<int32_t> before(parts, s);
  DBuf<uint8_t> part_kept(parts, s);
  for (int k = 0; k < 2; ++k) {
    CompactSide& d = sides.side[k];
    const size_t first = k ? size_t(sides.side[0].tiles) * kCompactWarps : 0;
    d.rows_at = row_bits + first * kCompactRounds;
    d.masks = masks.p + first * kCompactRounds;
    d.before = before.p + first;
    d.part_kept = part_kept.p + first;
  }
  // Every allocation before the first launch: one that fails leaves the bits zero.
  LookbackSpace w(size_t(tiles), s);
  const int rows_grid = grid_stride_blocks(std::max(sides.side[0].rows, sides.side[1].rows));
  GPP_LAUNCH(compact_mark_rows, rows_grid, kThreads, 0, s, sides);
  // Reads; the writes (12 nnz') are added to the launch's profile record once
  // the kept count is known.
  double bytes = 0.0;
  for (const CompactSide& d : sides.side)
    if (d.tiles) bytes += 12.0 * d.nnz + 4.0 * d.cols + 0.375 * d.nnz;
  const Report report = c.open_report(2);
  GPP_LAUNCH_BYTES(compact_tiles, bytes, std::min(tiles, kNumSMs * 5), kThreads, 0, s, sides, w.words, w.counters,
                   c.host_error, report);
  const int64_t record = profile_last();
  GPP_LAUNCH(compact_row_pointers, rows_grid, kThreads, 0, s, sides);
  const int64_t* kept = c.await(report);
  for (int k = 0; k < 2; ++k)
    if (sides.side[k].tiles) {
      out[k]->nnz = offset_t(kept[k]);
      profile_add_bytes(record, 12.0 * out[k]->nnz);
    }
}
}  // namespace

DevCsr compact_csr(const DevCsr& M, const int32_t* outer_map, int32_t outer_new, const int32_t* inner_map,
                   int32_t inner_new, cudaStream_t s) {
  CompactSides sides{};
  DevCsr out = compact_output(M, outer_map, outer_new, inner_map, inner_new, sides.side[0], s);
  compact_sides(sides, {&out, nullptr}, s);
  return out;
}

std::pair<DevCsr, DevCsr> compact_csr_pair(const DevCsr& A, const DevCsr& AT, const int32_t* row_map, int32_t rows_new,
                                           const int32_t* col_map, int32_t cols_new, cudaStream_t s) {
  CompactSides sides{};
  DevCsr a = compact_output(A, row_map, rows_new, col_map, cols_new, sides.side[0], s);
  DevCsr t = compact_output(AT, col_map, cols_new, row_map, rows_new, sides.side[1], s);
  compact_sides(sides, {&a, &t}, s);
  return {a, t};
}

DevCsr transpose_csr(const DevCsr& M, cudaStream_t s) {
  DevCsr t;
  t.rows = M.cols;
  t.cols = M.rows;
  t.nnz = M.nnz;
  t.ptr = dalloc<offset_t>(size_t(t.rows) + 1);
  if (M.nnz > 0) {
    t.idx = dalloc<int32_t>(size_t(M.nnz));
    t.val = dalloc<double>(size_t(M.nnz));
  }
  transpose_csr_into(M, t, s);
  return t;
}

void transpose_csr_into(const DevCsr& M, const DevCsr& t, cudaStream_t s) {
  // Entries ordered by column, each column in stored (row-major) order,
  // i.e. ascending rows (duplicates in stored order): the row-sorted CSR of
  // M^T.  Short columns (all at most kShortColumn long) use atomic slots and
  // a per-column sort of the positions; otherwise a stable radix sort.
  if (M.nnz == 0) {
    check(cudaMemsetAsync(t.ptr, 0, sizeof(offset_t) * (size_t(t.rows) + 1), s), "transpose empty");
    return;
  }
  DBuf<int32_t> cnt(size_t(t.rows) + 1, s);
  cnt.zero();
  const int g = grid_stride_blocks(M.nnz);
  GPP_LAUNCH(histogram, g, kThreads, 0, s, M.idx, M.nnz, cnt.p);
  exclusive_scan_i32(cnt.p, t.ptr, t.rows, s);
  DBuf<int32_t> pos(size_t(M.nnz), s), row(size_t(M.nnz), s);
  Status st;
  st.clear(1);
  GPP_LAUNCH(longest_count, grid_stride_blocks(t.rows), kThreads, 0, s, cnt.p, t.rows, st.d);
  if (st.read(1)[0] <= kShortColumn) {
    DBuf<int32_t> cursor(size_t(t.rows), s);
    check(cudaMemcpyAsync(cursor.p, t.ptr, sizeof(int32_t) * size_t(t.rows), cudaMemcpyDeviceToDevice, s),
          "transpose cursors");
    GPP_LAUNCH(place_positions, g, kThreads, 0, s, M.nnz, M.idx, cursor.p, pos.p);
    GPP_LAUNCH(order_columns, grid_stride_blocks(t.rows), kThreads, 0, s, t.rows, t.ptr, pos.p);
  } else {
    DBuf<uint64_t> keys(size_t(M.nnz), s);
    GPP_LAUNCH(transpose_keys, g, kThreads, 0, s, M.nnz, M.idx, keys.p, pos.p);
    radix_sort_pairs(keys.p, pos.p, M.nnz, s, bits_up_to(int64_t(M.cols) - 1));
  }
  GPP_LAUNCH(row_of_entry, std::max(1, std::min((M.rows + 7) / 8, kNumSMs * 16)), kThreads, 0, s, M.rows, M.ptr,
             row.p);
  GPP_LAUNCH(transpose_gather, g, kThreads, 0, s, M.nnz, pos.p, row.p, M.val, t.idx, t.val);
}

bool csr_structure_valid(const DevCsr& M, cudaStream_t s) {
  if (M.rows < 0 || M.cols < 0 || M.nnz < 0) return false;
  Status st;
  st.clear(1);
  GPP_LAUNCH(check_csr_structure, grid_stride_blocks(std::max<int64_t>(M.rows + 1, M.nnz)), kThreads, 0, s, M.rows,
             M.cols, M.nnz, M.ptr, M.idx, st.d);
  return st.read(1)[0] == 0;
}

bool rows_strictly_sorted(const DevCsr& M, cudaStream_t s) {
  if (M.rows <= 0 || M.nnz <= 1) return true;
  // A matrix does not change between materialisations, so the answer is kept
  // with its cached schedule.
  const RowSchedule& sch = stored_schedule(M);
  if (sch.sorted >= 0) return sch.sorted != 0;
  DBuf<int32_t> bad(1, s);
  bad.zero();
  GPP_LAUNCH(check_sorted, std::max(1, std::min((M.rows + 31) / 32, kNumSMs * 16)), kThreads, 0, s, M.rows, M.ptr,
             M.idx, bad.p);
  sch.sorted = read_scalar(bad.p) == 0 ? 1 : 0;
  return sch.sorted != 0;
}

void free_csr(DevCsr& M) {
  forget_schedule(M.ptr);
  dfree(M.ptr);
  dfree(M.idx);
  dfree(M.val);
  M = DevCsr{};
}

}  // namespace gpp

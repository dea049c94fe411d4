// Singleton-column rule: substitute out columns that appear in one live row.
//
// Reference: apply_rule_singleton_columns (cpp/src/presolve/rules/
// rule_singleton_columns.cu:1562-1827) with its kernels :459-1560.  The
// decisions are the reference's, evaluated against the unmodified plan:
//   * an activity cache per row holding a candidate (rows of live length
//     <= 1024 sum in stored order; longer rows give live rank k to thread
//     k mod 256 and reduce with a halving tree, :555-754);
//   * implied-free tests and the action choice (:756-903);
//   * one owner per row by atomicMin over keys that rank free eliminations
//     first, then the smallest column (:905-1018);
//   * staging (:1021-1073), the cost update c_k -= c_j a_ik / a_ij summed per
//     column in stored (row) order (:1075-1139), substitution and row-dual-
//     shift records in ascending row order (:459-508, :1191-1560).
// B200 layout of the work: the rule touches only the candidate columns, the
// rows that hold them and the columns of eliminated rows, through compacted
// work lists, instead of sweeping all of A / AT as the reference does.  The
// objective delta is the reference's canonical sum over the rule's entry
// domain.
#include <algorithm>
#include <climits>

#include "cleanup_probe.cuh"
#include "engine.cuh"
#include "live_visit.cuh"
#include "scan.cuh"
#include "sort.hpp"

namespace gpp {

namespace {

enum : uint8_t {
  kNone = 0, kSetRowSide = 1, kTightenLhs = 2, kTightenRhs = 3,
  kEliminateFree = 4, kEliminateFreeAbove = 5, kEliminateFreeBelow = 6
};
// Row kinds after staging (only rows in the winner list carry one).
enum : uint8_t { kRowElimKept = 1, kRowElimDeleted = 2, kRowDualShift = 3 };

constexpr int kUnclaimed = kUnclaimedRow;
constexpr int kClaimed = INT_MAX - 1;   // row holds a candidate, no owner yet

// Status words.
enum { kStUnbounded = 0, kStCand = 1, kStRows = 2, kStLong = 3, kStWin = 4, kStElim = 5, kStSide = 6,
       kStTouched = 7, kStWords = kSingletonWords };

__device__ __forceinline__ bool direct_unbounded(double cj, double a, double lhs, double rhs, double lb, double ub,
                                                 double zt) {
  // _singleton_column_direct_unbounded (rule_singleton_columns.cu:516-527).
  return (cj > zt && a > zt && !isfinite(lhs) && !isfinite(lb)) ||
         (cj > zt && a < -zt && !isfinite(rhs) && !isfinite(lb)) ||
         (cj < -zt && a < -zt && !isfinite(lhs) && !isfinite(ub)) ||
         (cj < -zt && a > zt && !isfinite(rhs) && !isfinite(ub));
}

// What the rule's kernels read, and the lists and scratch that one writes and
// the next reads (no `__restrict__`: the fused kernel runs all four).
struct ScArgs {
  int n, m, row_blocks, long_blocks;
  const uint8_t* singleton;
  const int32_t* srow;
  const double* sval;
  const int32_t* row_nnz;
  const double *c, *l, *u;
  const double2* lu;
  const offset_t* ptr;
  const int32_t* idx;
  const double* val;
  double tol, zero_tol;
  double *AL, *AU;
  uint8_t *keep_row, *keep_col;
  int32_t *owner, *cand, *rows, *long_rows, *st, *winners;
  double *fmin, *fmax;
  int4* counts;
  uint8_t *invalid, *action, *kind;
  double *side, *contrib_val;
  int64_t* contrib_idx;
};

// Candidates (:905-940): kept singleton column in a kept row with another
// live entry and |a| > zero_tol.  Directly unbounded candidates only raise the
// flag.  The first candidate of a row claims it for the cache and stage lists.
// A block takes 1,024 columns at a time, four to a thread: blocks without a
// candidate go on after one barrier, the others rank all three lists with one
// block scan.  (A form that appended each list for 256 columns stood at its nine
// barriers with DRAM at 6% of its rate, 94 us over 5M columns.)
__device__ __forceinline__ void sc_candidates_part(const ScArgs& g) {
  constexpr int kPer = 4;
  constexpr int kField = 20;   // bits of a list's count, at most 1,024 a block
  __shared__ unsigned long long warp_sums[kThreads / 32];
  __shared__ int bases[3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double zero_tol = g.zero_tol;
  for (int64_t base = int64_t(blockIdx.x) * (kThreads * kPer); base < g.n; base += int64_t(gridDim.x) * (kThreads * kPer)) {
    int row[kPer];
    double a[kPer];
    bool cand[kPer];
    unsigned take = 0, claim = 0, is_long = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int64_t j = base + k * kThreads + threadIdx.x;
      cand[k] = j < g.n && (g.keep_col[j] != 0) & (g.singleton[j] != 0);
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int64_t j = base + k * kThreads + threadIdx.x;
      row[k] = cand[k] ? g.srow[j] : -1;
      a[k] = cand[k] ? g.sval[j] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int64_t j = base + k * kThreads + threadIdx.x;
      const int r = row[k];
      if (!(r >= 0 && r < g.m) || fabs(a[k]) <= zero_tol || !g.keep_row[r]) continue;
      const int len = g.row_nnz[r];
      if (len <= 1) continue;
      if (direct_unbounded(g.c[j], a[k], g.AL[r], g.AU[r], g.l[j], g.u[j], zero_tol)) {
        atomicOr(g.st + kStUnbounded, 1);
        continue;
      }
      take |= 1u << k;
      if (atomicCAS(g.owner + r, kUnclaimed, kClaimed) == kUnclaimed) {
        claim |= 1u << k;
        if (len > kLongRow) is_long |= 1u << k;
      }
    }
    if (!__syncthreads_or(take)) continue;
    const unsigned long long own = (unsigned long long)__popc(take) | (unsigned long long)__popc(claim) << kField |
                                   (unsigned long long)__popc(is_long) << 2 * kField;
    unsigned long long upto = own;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned long long v = __shfl_up_sync(0xffffffffu, upto, off);
      if (lane >= off) upto += v;
    }
    if (lane == 31) warp_sums[warp] = upto;
    __syncthreads();
    unsigned long long before = upto - own, all = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
      before += w < warp ? warp_sums[w] : 0ull;
      all += warp_sums[w];
    }
    const unsigned long long field = (1ull << kField) - 1;
    if (threadIdx.x < 3) {
      const int count = int(all >> (kField * threadIdx.x) & field);
      bases[threadIdx.x] = count ? atomicAdd(g.st + kStCand + threadIdx.x, count) : 0;
    }
    __syncthreads();
    int at[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) at[q] = bases[q] + int(before >> (kField * q) & field);
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      if (take >> k & 1u) g.cand[at[0]++] = int(base + k * kThreads + threadIdx.x);
      if (claim >> k & 1u) g.rows[at[1]++] = row[k];
      if (is_long >> k & 1u) g.long_rows[at[2]++] = row[k];
    }
  }
}
static_assert(kStRows == kStCand + 1 && kStLong == kStCand + 2, "one counter per list");
__global__ void __launch_bounds__(kThreads) sc_candidates(ScArgs g, const int32_t* gate) {
  after_previous_kernel();
  if (gate && *gate) return;   // the lists stay empty for the kernels behind
  sc_candidates_part(g);
}

struct RowCache {
  double fmin, fmax;
  int min_neg, min_pos, max_neg, max_pos;
  int invalid;
};

__device__ __forceinline__ void cache_term(RowCache& r, double a, double lj, double uj) {
  const double tmin = a >= 0.0 ? a * lj : a * uj;
  const double tmax = a >= 0.0 ? a * uj : a * lj;
  if (isnan(tmin) || isnan(tmax)) { r.invalid = 1; return; }
  if (isinf(tmin)) { if (tmin < 0.0) ++r.min_neg; else ++r.min_pos; } else { r.fmin += tmin; }
  if (isinf(tmax)) { if (tmax < 0.0) ++r.max_neg; else ++r.max_pos; } else { r.fmax += tmax; }
}

struct CacheOut {
  double *fmin, *fmax;
  int4* counts;
  uint8_t* invalid;
  __device__ void store(int row, const RowCache& r) const {
    fmin[row] = r.fmin;
    fmax[row] = r.fmax;
    counts[row] = make_int4(r.min_neg, r.min_pos, r.max_neg, r.max_pos);
    invalid[row] = uint8_t(r.invalid);
  }
};

// A column's bounds for the cache: the packed records where the plan holds
// them as it stands (one access of 16 bytes), the mask and both bounds else.
template <bool kPacked>
struct CacheBounds {
  const double2* lu;
  const uint8_t* keep_col;
  const double *l, *u;
  __device__ __forceinline__ bool get(int col, double2& b) const {
    if constexpr (kPacked) {
      b = lu[col];
      return !removed_column(b);
    } else {
      if (!keep_col[col]) return false;
      b = make_double2(l[col], u[col]);
      return true;
    }
  }
};

// _kernel_singleton_row_activity_cache (:555-614) for rows of live length
// <= 1024.  The reference's sequential loop skips a NaN term entirely, counts
// an infinite term and adds a finite one; the counts and the NaN flag are
// order-free, so they come from ballots (where a row of the warp has such a
// term), and the finite sums are formed in stored order, from shared memory, by
// one lane each, for as many steps as the warp's longest row has (a chain of 32
// shuffles over all lanes kept the shuffle unit busy: 162 us at the 29.8M-nnz
// LP).  A
// skipped term enters the chain as +0.0, which is exact: a sum that starts at
// +0.0 never becomes -0.0 in round-to-nearest, and x + (+0.0) == x for every
// other x.  Rows of at most 32 stored entries (nearly all) take eight lanes
// each, four rows per warp, with all of a row's loads issued before its
// chain; longer rows take a whole warp, 32 entries at a time.
template <bool kPacked>
__device__ void sc_cache_rows(int blocks, const int32_t* rows, const int32_t* st,
                              const int32_t* __restrict__ row_nnz, const offset_t* __restrict__ ptr,
                              const int32_t* __restrict__ idx, const double* __restrict__ val,
                              CacheBounds<kPacked> bounds, CacheOut out) {
  __shared__ double terms[kThreads / 32][2][4][33];   // by warp, sum and row; a row's padded by one
  const int count = st[kStRows];
  const int lane = threadIdx.x & 31, grp = lane >> 3, gl = lane & 7, warp = threadIdx.x >> 5;
  const int warps = blocks * (blockDim.x >> 5);
  const auto group_bits = [&](bool v) { return (__ballot_sync(0xffffffffu, v) >> (grp * 8)) & 0xffu; };
  const auto whole_row = [&](int row) {
    RowCache r{0.0, 0.0, 0, 0, 0, 0, 0};
    const offset_t end = ptr[row + 1];
    for (offset_t chunk = ptr[row]; chunk < end; chunk += 32) {
      const offset_t p = chunk + lane;
      double tmin = 0.0, tmax = 0.0;
      bool live = false;
      if (p < end) {
        const int col = __ldcs(idx + p);
        double2 b;
        live = bounds.get(col, b);
        if (live) {
          const double a = __ldcs(val + p);
          tmin = a >= 0.0 ? a * b.x : a * b.y;
          tmax = a >= 0.0 ? a * b.y : a * b.x;
        }
      }
      const bool nan = live && (isnan(tmin) || isnan(tmax));
      const bool counted = live && !nan;
      r.invalid |= __any_sync(0xffffffffu, nan);
      r.min_neg += __popc(__ballot_sync(0xffffffffu, counted && isinf(tmin) && tmin < 0.0));
      r.min_pos += __popc(__ballot_sync(0xffffffffu, counted && isinf(tmin) && tmin > 0.0));
      r.max_neg += __popc(__ballot_sync(0xffffffffu, counted && isinf(tmax) && tmax < 0.0));
      r.max_pos += __popc(__ballot_sync(0xffffffffu, counted && isinf(tmax) && tmax > 0.0));
      const double fmin_term = counted && isfinite(tmin) ? tmin : 0.0;
      const double fmax_term = counted && isfinite(tmax) ? tmax : 0.0;
      const int n = int(min(offset_t(32), end - chunk));
      for (int k = 0; k < n; ++k) {
        r.fmin += __shfl_sync(0xffffffffu, fmin_term, k);
        r.fmax += __shfl_sync(0xffffffffu, fmax_term, k);
      }
    }
    if (lane == 0) out.store(row, r);
  };
  // Row ids two iterations ahead and row pointers and lengths one ahead, so
  // an iteration's critical path starts at its entries.
  const int step = warps * 4;
  const int w_first = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 4 + grp;
  int row_next = w_first < count ? rows[w_first] : 0;
  int row_after = w_first + step < count ? rows[w_first + step] : 0;
  int len_next = w_first < count ? row_nnz[row_next] : 0;
  offset_t first_next = w_first < count ? ptr[row_next] : 0, end_next = w_first < count ? ptr[row_next + 1] : 0;
  for (int w0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 4; w0 < count; w0 += step) {
    const int w = w0 + grp;
    const int row = row_next;
    const bool take = w < count && len_next <= kLongRow;
    const offset_t first = take ? first_next : 0, end = take ? end_next : 0;
    row_next = row_after;
    const bool more = w + step < count;
    len_next = more ? row_nnz[row_next] : 0;
    first_next = more ? ptr[row_next] : 0;
    end_next = more ? ptr[row_next + 1] : 0;
    row_after = w + 2 * step < count ? rows[w + 2 * step] : 0;
    const bool grouped = take && end - first <= 32;
    const offset_t stop = grouped ? end : first;
    int col[4];
    double a[4], lj[4], uj[4];
    bool live[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const offset_t p = first + gl + 8 * j;
      col[j] = p < stop ? __ldcs(idx + p) : -1;
      a[j] = p < stop ? __ldcs(val + p) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      double2 b = make_double2(0.0, 0.0);
      live[j] = col[j] >= 0 && bounds.get(col[j], b);
      lj[j] = b.x;
      uj[j] = b.y;
    }
    RowCache r{0.0, 0.0, 0, 0, 0, 0, 0};
    const int steps = __reduce_max_sync(0xffffffffu, int(stop - first));   // of the warp's longest row
    bool odd = false;   // a NaN or infinite term in the warp's rows
    double tmin[4], tmax[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      tmin[j] = live[j] ? (a[j] >= 0.0 ? a[j] * lj[j] : a[j] * uj[j]) : 0.0;
      tmax[j] = live[j] ? (a[j] >= 0.0 ? a[j] * uj[j] : a[j] * lj[j]) : 0.0;
      odd = odd || !isfinite(tmin[j]) || !isfinite(tmax[j]);
      if (8 * j < steps) {
        const bool counted = !isnan(tmin[j]) && !isnan(tmax[j]);
        terms[warp][0][grp][gl + 8 * j] = counted && isfinite(tmin[j]) ? tmin[j] : 0.0;
        terms[warp][1][grp][gl + 8 * j] = counted && isfinite(tmax[j]) ? tmax[j] : 0.0;
      }
    }
    if (__any_sync(0xffffffffu, odd)) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool nan = isnan(tmin[j]) || isnan(tmax[j]);
        r.invalid |= group_bits(nan) != 0;
        r.min_neg += __popc(group_bits(!nan && isinf(tmin[j]) && tmin[j] < 0.0));
        r.min_pos += __popc(group_bits(!nan && isinf(tmin[j]) && tmin[j] > 0.0));
        r.max_neg += __popc(group_bits(!nan && isinf(tmax[j]) && tmax[j] < 0.0));
        r.max_pos += __popc(group_bits(!nan && isinf(tmax[j]) && tmax[j] > 0.0));
      }
    }
    __syncwarp();
    double sum = 0.0;
    if (gl < 2) {   // lane 0 of a row folds its minimum, lane 1 its maximum
      const double* term = terms[warp][gl][grp];
      for (int k = 0; k < steps; k += 8)
#pragma unroll
        for (int q = 0; q < 8; ++q) sum += term[k + q];
    }
    __syncwarp();
    r.fmin = sum;
    r.fmax = __shfl_down_sync(0xffffffffu, sum, 1);
    if (grouped && gl == 0) out.store(row, r);
    unsigned rest = __ballot_sync(0xffffffffu, take && !grouped && gl == 0);
    while (rest) {
      const int src = __ffs(rest) - 1;
      rest &= rest - 1;
      whole_row(__shfl_sync(0xffffffffu, row, src));
    }
  }
}

// _kernel_singleton_long_row_activity_cache (:642-754): block per row; live
// rank k goes to thread k mod 256, then a shared-memory halving tree.
template <bool kPacked>
__device__ void sc_cache_long(int block, int blocks, const int32_t* long_rows,
                              const int32_t* st, const int32_t* __restrict__ row_nnz,
                              const offset_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                              const double* __restrict__ val, CacheBounds<kPacked> bounds, CacheOut out) {
  __shared__ int slots[kThreads];
  __shared__ int warp_counts[8];
  __shared__ double s_min[kThreads], s_max[kThreads];
  __shared__ int s_cnt[5][kThreads];
  const int count = st[kStLong];
  const int t = threadIdx.x;
  for (int q = block; q < count; q += blocks) {
    const int row = long_rows[q];
    const offset_t first = ptr[row], last = ptr[row + 1];
    const uint8_t* mask = row_nnz[row] != int(last - first) ? bounds.keep_col : nullptr;
    RowCache r{0.0, 0.0, 0, 0, 0, 0, 0};
    live_visit<kThreads>(first, last, idx, mask, slots, warp_counts, [&](offset_t p) {
      const int col = idx[p];
      double2 b;
      if (bounds.get(col, b)) cache_term(r, val[p], b.x, b.y);
    });
    s_min[t] = r.fmin;
    s_max[t] = r.fmax;
    s_cnt[0][t] = r.min_neg; s_cnt[1][t] = r.min_pos; s_cnt[2][t] = r.max_neg; s_cnt[3][t] = r.max_pos;
    s_cnt[4][t] = r.invalid;
    __syncthreads();
    for (int h = kThreads / 2; h > 0; h >>= 1) {
      if (t < h) {
        s_min[t] += s_min[t + h];
        s_max[t] += s_max[t + h];
        for (int k = 0; k < 4; ++k) s_cnt[k][t] += s_cnt[k][t + h];
        s_cnt[4][t] |= s_cnt[4][t + h];
      }
      __syncthreads();
    }
    if (t == 0)
      out.store(row, RowCache{s_min[0], s_max[0], s_cnt[0][0], s_cnt[1][0], s_cnt[2][0], s_cnt[3][0], s_cnt[4][0]});
    __syncthreads();
  }
}

// Both roles in one launch: the first `row_blocks` blocks take the claimed
// rows of up to kLongRow live entries, the rest the long ones.  The grid does
// not know their numbers (the rule asks the host once, at its end); blocks
// without rows return at once.
template <bool kPacked>
__device__ __forceinline__ CacheBounds<kPacked> cache_bounds(const ScArgs& g) {
  return CacheBounds<kPacked>{g.lu, g.keep_col, g.l, g.u};
}
template <bool kPacked>
__global__ void __launch_bounds__(kThreads) sc_cache(ScArgs g) {
  after_previous_kernel();
  const CacheOut out{g.fmin, g.fmax, g.counts, g.invalid};
  if (int(blockIdx.x) < g.row_blocks)
    sc_cache_rows(g.row_blocks, g.rows, g.st, g.row_nnz, g.ptr, g.idx, g.val, cache_bounds<kPacked>(g), out);
  else
    sc_cache_long(int(blockIdx.x) - g.row_blocks, g.long_blocks, g.long_rows, g.st, g.row_nnz, g.ptr, g.idx, g.val,
                  cache_bounds<kPacked>(g), out);
}

// Propose (:905-1018) over the candidate list.
__device__ __forceinline__ void sc_propose_part(const ScArgs& g) {
  const int32_t* const st = g.st;
  const double tol = g.tol, zero_tol = g.zero_tol;
  const int count = st[kStCand];
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x) {
    const int j = g.cand[q];
    const int row = g.srow[j];
    const double a = g.sval[j];
    const double lj = g.l[j], uj = g.u[j], cj = g.c[j];
    // _singleton_column_activity_bounds_from_cache (:756-816).
    if (g.invalid[row]) continue;
    const double tmin = a >= 0.0 ? a * lj : a * uj;
    const double tmax = a >= 0.0 ? a * uj : a * lj;
    if (isnan(tmin) || isnan(tmax)) continue;
    int4 k = g.counts[row];
    double vmin = g.fmin[row], vmax = g.fmax[row];
    if (isinf(tmin)) { if (tmin < 0.0) --k.x; else --k.y; } else { vmin -= tmin; }
    if (isinf(tmax)) { if (tmax < 0.0) --k.z; else --k.w; } else { vmax -= tmax; }
    if (k.x < 0 || k.y < 0 || k.z < 0 || k.w < 0 || (k.x > 0 && k.y > 0) || (k.z > 0 && k.w > 0)) continue;
    const double rmin = k.x > 0 ? -INFINITY : (k.y > 0 ? INFINITY : vmin);
    const double rmax = k.z > 0 ? -INFINITY : (k.w > 0 ? INFINITY : vmax);
    if (isnan(rmin) || isnan(rmax)) continue;
    const double lhs = g.AL[row], rhs = g.AU[row];
    uint8_t act = kNone;
    double sd = 0.0;
    if (isfinite(lhs) && isfinite(rhs) && fabs(lhs - rhs) <= tol) {
      const double x1 = (rhs - rmin) / a, x2 = (rhs - rmax) / a;
      const double ilb = fmin(x1, x2), iub = fmax(x1, x2);
      const bool above = !isfinite(uj) || iub <= uj + tol;
      const bool below = !isfinite(lj) || ilb >= lj - tol;
      if (!(above || below)) continue;
      act = above && below ? kEliminateFree : (above ? kEliminateFreeAbove : kEliminateFreeBelow);
      sd = rhs;
    } else {
      // _singleton_column_implied_free_from_above / _below (:818-854).
      bool above = true, below = true;
      if (isfinite(uj)) {
        double implied = INFINITY;
        if (a > 0.0 && isfinite(rhs)) implied = (rhs - rmin) / a;
        else if (a < 0.0 && isfinite(lhs)) implied = (lhs - rmax) / a;
        above = implied <= uj + tol;
      }
      if (isfinite(lj)) {
        double implied = -INFINITY;
        if (a > 0.0 && isfinite(lhs)) implied = (lhs - rmax) / a;
        else if (a < 0.0 && isfinite(rhs)) implied = (rhs - rmin) / a;
        below = implied >= lj - tol;
      }
      // _singleton_column_active_side / _ineq_action (:856-903).
      if (above && below) {
        if ((cj > zero_tol && a > 0.0) || (cj < -zero_tol && a < 0.0)) sd = lhs;
        else if ((cj > zero_tol && a < 0.0) || (cj < -zero_tol && a > 0.0)) sd = rhs;
        else sd = isfinite(lhs) ? lhs : rhs;
        if (!isfinite(sd)) continue;
        act = kSetRowSide;
      } else if (((cj < -zero_tol && a > 0.0 && above) || (cj > zero_tol && a < 0.0 && below)) && isfinite(rhs)) {
        act = kTightenLhs;
        sd = rhs;
      } else if (((cj > zero_tol && a > 0.0 && below) || (cj < -zero_tol && a < 0.0 && above)) && isfinite(lhs)) {
        act = kTightenRhs;
        sd = lhs;
      } else {
        continue;
      }
    }
    g.action[j] = act;
    g.side[j] = sd;
    atomicMin(g.owner + row, act == kEliminateFree ? j - INT_MAX : j);
  }
}
__global__ void __launch_bounds__(kThreads) sc_propose(ScArgs g) {
  after_previous_kernel();
  sc_propose_part(g);
}

// Stage + commit (:1021-1073, :1157-1189) over the claimed rows.  Every read
// is of the owner's own row and column, so the plan is updated in place; the
// row keeps its owner in `owner` only when the owner column is eliminated.
__device__ __forceinline__ void sc_stage_part(const ScArgs& g) {
  int32_t* const st = g.st;
  const int n = g.n;
  const double tol = g.tol;
  // An unbounded candidate ends the rule with the plan as it was.
  const int count = st[kStUnbounded] ? 0 : st[kStRows];
  const int stride = gridDim.x * blockDim.x;
  const int top = (count + stride - 1) / stride * stride;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < top; q += stride) {
    int row = -1, j = -1;
    uint8_t k = 0;
    double contrib = 0.0;
    if (q < count) {
      row = g.rows[q];
      const int key = g.owner[row];
      j = key < 0 ? key + INT_MAX : key;
      if (j >= 0 && j < n) {
        const uint8_t act = g.action[j];
        const double lhs = g.AL[row], rhs = g.AU[row];
        if (act == kEliminateFree || act == kEliminateFreeAbove || act == kEliminateFreeBelow) {
          const double a = g.sval[j];
          contrib = g.c[j] * rhs / a;
          if (act == kEliminateFree) {
            g.keep_row[row] = 0;
            k = kRowElimDeleted;
          } else {
            const bool above = act == kEliminateFreeAbove;
            const double bound = above ? g.l[j] : g.u[j];
            const bool keep_lower = above ? a < 0.0 : a > 0.0;
            const double shifted = rhs - a * bound;
            if (keep_lower) { g.AL[row] = shifted; g.AU[row] = INFINITY; }
            else { g.AL[row] = -INFINITY; g.AU[row] = shifted; }
            k = kRowElimKept;
          }
          g.keep_col[j] = 0;
          g.owner[row] = j;
        } else {
          bool lo = false, hi = false;
          const double sd = g.side[j];
          if (act == kSetRowSide) {
            lo = !isfinite(lhs) || fabs(lhs - sd) > tol;
            hi = !isfinite(rhs) || fabs(rhs - sd) > tol;
            g.AL[row] = sd;
            g.AU[row] = sd;
          } else if (act == kTightenLhs) {
            lo = true;
            g.AL[row] = rhs;
          } else if (act == kTightenRhs) {
            hi = true;
            g.AU[row] = lhs;
          }
          atomicOr(st + kStSide, 1);
          if (lo || hi) k = kRowDualShift;
          g.owner[row] = kUnclaimed;
        }
      } else {
        g.owner[row] = kUnclaimed;
      }
      if (k) g.kind[row] = k;
    }
    const bool elim = k == kRowElimKept || k == kRowElimDeleted;
    const int pe = block_append(st + kStElim, elim);
    if (elim) { g.contrib_idx[pe] = j; g.contrib_val[pe] = contrib; }
    const int pw = block_append(st + kStWin, k != 0);
    if (k) g.winners[pw] = row;
  }
}
__global__ void __launch_bounds__(kThreads) sc_stage(ScArgs g, Report report) {
  after_previous_kernel();
  sc_stage_part(g);
  post_report(report);
}

// Probe and rule as one cluster, for models whose kernels are shorter than
// their launches: the cluster's barrier stands where a launch did.  Its blocks
// are scheduled together, so nothing spins.  At 2,000 x 5,000 the five launches
// and two waits took about 52 us.
template <bool kPacked>
__global__ void __cluster_dims__(kSmallCluster, 1, 1) __launch_bounds__(kThreads)
probe_and_singleton_columns(ProbeArgs probe, ScArgs g, Report report) {
  after_previous_kernel();
  if (blockIdx.x == 0 && threadIdx.x <= kSingletonWords) g.st[threadIdx.x] = 0;
  const uint32_t found = probe_part(probe);
  cluster_barrier();   // words and owners are cleared
  Report probed = report;
  probed.words = g.st + kSingletonWords;
  gather_flags(probed, found);
  cluster_barrier();
  if (*static_cast<volatile int32_t*>(probed.words) == 0) {   // the same in every block
    sc_candidates_part(g);
    cluster_barrier();
    const CacheOut out{g.fmin, g.fmax, g.counts, g.invalid};
    sc_cache_rows(kSmallCluster, g.rows, g.st, g.row_nnz, g.ptr, g.idx, g.val, cache_bounds<kPacked>(g), out);
    sc_cache_long(int(blockIdx.x), kSmallCluster, g.long_rows, g.st, g.row_nnz, g.ptr, g.idx, g.val,
                  cache_bounds<kPacked>(g), out);
    cluster_barrier();
    sc_propose_part(g);
    cluster_barrier();
    sc_stage_part(g);
  }
  post_report(report);
}

// Columns whose cost changes: the live columns of eliminated rows, each
// claimed once through a byte flag.
__global__ void sc_touch(const int32_t* __restrict__ winners, const int32_t* __restrict__ st,
                         const uint8_t* __restrict__ kind, const offset_t* __restrict__ ptr,
                         const int32_t* __restrict__ idx, const uint8_t* __restrict__ keep_col,
                         uint32_t* __restrict__ claimed, int32_t* __restrict__ touched, int32_t* st_w) {
  after_previous_kernel();
  const int count = st[kStWin];
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  for (int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < count; w += warps) {
    const int row = winners[w];
    if (kind[row] == kRowDualShift) continue;
    for (offset_t chunk = ptr[row]; chunk < ptr[row + 1]; chunk += 32) {
      const offset_t p = chunk + lane;
      bool take = false;
      int col = 0;
      if (p < ptr[row + 1]) {
        col = idx[p];
        if (keep_col[col]) {
          const uint32_t bit = 1u << (col & 31);
          take = (atomicOr(claimed + (col >> 5), bit) & bit) == 0;
        }
      }
      const int pos = warp_append(st_w + kStTouched, take);
      if (take) touched[pos] = col;
    }
  }
}

// _kernel_apply_singleton_objective_updates_deterministic (:1075-1104): for a
// touched column, c += -(c_o * a / a_o) over its stored entries whose row is
// eliminated by owner o, added in stored order.  Each column belongs to one
// warp and the owners' costs are never touched, so c is updated in place.
__global__ void sc_cost(const int32_t* __restrict__ touched, const int32_t* __restrict__ st, int n,
                        const offset_t* __restrict__ tptr, const int32_t* __restrict__ tidx,
                        const double* __restrict__ tval, const int32_t* __restrict__ owner,
                        const double* __restrict__ sval, double* __restrict__ c) {
  after_previous_kernel();
  const int count = st[kStTouched];
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  for (int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < count; w += warps) {
    const int col = touched[w];
    double updated = c[col];
    for (offset_t chunk = tptr[col]; chunk < tptr[col + 1]; chunk += 32) {
      const offset_t p = chunk + lane;
      double term = 0.0;
      bool has = false;
      if (p < tptr[col + 1]) {
        const int o = owner[tidx[p]];
        if (o >= 0 && o < n) {
          has = true;
          term = -(c[o] * tval[p] / sval[o]);
        }
      }
      const unsigned hv = __ballot_sync(0xffffffffu, has);
      for (int k = 0; k < 32; ++k) {
        const double v = __shfl_sync(0xffffffffu, term, k);
        if (hv >> k & 1u) updated += v;
      }
    }
    if (lane == 0) c[col] = updated;
  }
}

// Substitution record sizes (:1191-1284): pivot and live support of each
// eliminated row, in ascending row order.
__global__ void sc_sub_sizes(const int32_t* __restrict__ sorted_rows, int count, const int32_t* __restrict__ owner,
                             const offset_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                             const double* __restrict__ val, const uint8_t* __restrict__ keep_col, double zero_tol,
                             int32_t* __restrict__ sel, int64_t* __restrict__ support) {
  after_previous_kernel();
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  for (int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < count; w += warps) {
    const int row = sorted_rows[w];
    const int col = owner[row];
    int cnt = 0;
    double pivot = 0.0;
    for (offset_t p = ptr[row] + lane; p < ptr[row + 1]; p += 32) {
      const int rc = idx[p];
      if (rc == col) pivot = val[p];
      else if (keep_col[rc]) ++cnt;
    }
    for (int off = 16; off > 0; off >>= 1) {
      cnt += __shfl_down_sync(0xffffffffu, cnt, off);
      const double other = __shfl_down_sync(0xffffffffu, pivot, off);
      if (other != 0.0) pivot = other;
    }
    if (lane == 0) {
      const bool ok = !(fabs(pivot) <= zero_tol);
      sel[w] = ok ? 1 : 0;
      support[w] = ok ? cnt : 0;
    }
  }
}

// SingletonColumnSubstitution records: indices [col, row, count, support...],
// values [pivot, side, l, u, c, row_deleted, coefficients...]; the support
// keeps the stored order (warp ballot compaction).
__global__ void sc_sub_pack(const int32_t* __restrict__ sorted_rows, int count, const int32_t* __restrict__ owner,
                            const uint8_t* __restrict__ kind, const int32_t* __restrict__ sel,
                            const int32_t* __restrict__ rec, const int64_t* __restrict__ spos,
                            const offset_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                            const double* __restrict__ val, const uint8_t* __restrict__ keep_col,
                            const double* __restrict__ side, const double* __restrict__ c,
                            const double* __restrict__ l, const double* __restrict__ u, int32_t* __restrict__ types,
                            int64_t* __restrict__ is, int64_t* __restrict__ vs, int32_t* __restrict__ oidx,
                            double* __restrict__ oval) {
  after_previous_kernel();
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  for (int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < count; w += warps) {
    if (!sel[w]) continue;
    const int row = sorted_rows[w];
    const int col = owner[row];
    const int64_t r = rec[w];
    const int64_t s0 = spos[w], s1 = spos[w + 1];
    const int64_t i0 = 3 * r + s0, v0 = 6 * r + s0;
    if (lane == 0) {
      if (r == 0) { is[0] = 0; vs[0] = 0; }
      types[r] = 2;  // SingletonColumnSubstitution
      is[r + 1] = 3 * (r + 1) + s1;
      vs[r + 1] = 6 * (r + 1) + s1;
      oidx[i0] = col;
      oidx[i0 + 1] = row;
      oidx[i0 + 2] = int32_t(s1 - s0);
      oval[v0 + 1] = side[col];
      oval[v0 + 2] = l[col];
      oval[v0 + 3] = u[col];
      oval[v0 + 4] = c[col];
      oval[v0 + 5] = kind[row] == kRowElimDeleted ? 1.0 : 0.0;
    }
    int64_t out = 0;
    for (offset_t chunk = ptr[row]; chunk < ptr[row + 1]; chunk += 32) {
      const offset_t p = chunk + lane;
      bool take = false;
      int rc = -1;
      double a = 0.0;
      if (p < ptr[row + 1]) {
        rc = idx[p];
        a = val[p];
        if (rc == col) oval[v0] = a;
        else take = keep_col[rc] != 0;
      }
      const unsigned mask = __ballot_sync(0xffffffffu, take);
      if (take) {
        const int64_t o = out + __popc(mask & ((1u << lane) - 1u));
        oidx[i0 + 3 + o] = rc;
        oval[v0 + 6 + o] = a;
      }
      out += __popc(mask);
    }
  }
}

// RowDualShift records (:459-508): index [row], value 0.0.
__global__ void sc_shift_pack(const int32_t* __restrict__ sorted_rows, int count, int32_t* __restrict__ types,
                              int64_t* __restrict__ is, int64_t* __restrict__ vs, int32_t* __restrict__ oidx,
                              double* __restrict__ oval) {
  after_previous_kernel();
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < count; r += gridDim.x * blockDim.x) {
    if (r == 0) { is[0] = 0; vs[0] = 0; }
    types[r] = 10;  // RowDualShift
    is[r + 1] = r + 1;
    vs[r + 1] = r + 1;
    oidx[r] = sorted_rows[r];
    oval[r] = 0.0;
  }
}

// Unclaimed owners and zeroed status words.
__global__ void sc_start(int32_t* p, int n, int32_t v, int32_t* __restrict__ st) {
  after_previous_kernel();
  if (blockIdx.x == 0 && threadIdx.x < kStWords) st[threadIdx.x] = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = v;
}

// The objective contributions as a dense vector for the canonical sum.
__global__ void sc_scatter_contrib(int count, const int64_t* __restrict__ idx, const double* __restrict__ val,
                                   double* __restrict__ dense) {
  after_previous_kernel();
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x) dense[idx[q]] = val[q];
}

// Sort key: substitution rows first, then dual-shift rows, each ascending.
__global__ void sc_winner_keys(const int32_t* __restrict__ winners, int count, const uint8_t* __restrict__ kind,
                               uint64_t* __restrict__ keys, int32_t* __restrict__ vals) {
  after_previous_kernel();
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x) {
    const int row = winners[q];
    keys[q] = (uint64_t(kind[row] == kRowDualShift ? 1 : 0) << 32) | uint32_t(row);
    vals[q] = row;
  }
}

}  // namespace

namespace {
ScArgs singleton_args(SingletonTest& t, Plan& plan, const WorkingLp& lp, const Stats& stats, const gpp_params& p) {
  const int m = lp.m(), n = lp.n();
  auto s = ctx().stream;
  const int claims = std::min(m, n);   // at most: one per row and per candidate
  t.cand.alloc(size_t(n), s);
  t.rows.alloc(size_t(m), s);
  t.long_rows.alloc(size_t(m), s);
  t.winners.alloc(size_t(claims), s);
  t.fmin.alloc(size_t(m), s);
  t.fmax.alloc(size_t(m), s);
  t.side.alloc(size_t(n), s);
  t.contrib_val.alloc(size_t(claims), s);
  t.counts.alloc(size_t(m), s);
  t.invalid.alloc(size_t(m), s);
  t.action.alloc(size_t(n), s);
  t.kind.alloc(size_t(m), s);
  t.contrib_idx.alloc(size_t(claims), s);
  ScArgs g{};
  g.n = n;
  g.m = m;
  g.row_blocks = std::max(1, std::min((claims + 31) / 32, kNumSMs * 16));
  g.long_blocks = std::max(1, std::min(kNumSMs * 4, int(lp.A.nnz / kLongRow)));
  g.singleton = stats.singleton_col.p;
  g.srow = stats.scol_row.p;
  g.sval = stats.scol_val.p;
  g.row_nnz = stats.row_nnz.p;
  g.c = plan.c.p;
  g.l = plan.l.p;
  g.u = plan.u.p;
  g.lu = plan.lu.p;
  g.ptr = lp.A.ptr;
  g.idx = lp.A.idx;
  g.val = lp.A.val;
  g.tol = p.bound_tol;
  g.zero_tol = p.zero_tol;
  g.AL = plan.AL.p;
  g.AU = plan.AU.p;
  g.keep_row = plan.keep_row.p;
  g.keep_col = plan.keep_col.p;
  g.owner = plan.sc_owner.p;
  g.st = plan.sc_words.p;
  g.cand = t.cand.p;
  g.rows = t.rows.p;
  g.long_rows = t.long_rows.p;
  g.winners = t.winners.p;
  g.fmin = t.fmin.p;
  g.fmax = t.fmax.p;
  g.counts = t.counts.p;
  g.invalid = t.invalid.p;
  g.action = t.action.p;
  g.kind = t.kind.p;
  g.side = t.side.p;
  g.contrib_val = t.contrib_val.p;
  g.contrib_idx = t.contrib_idx.p;
  return g;
}
}  // namespace

void ask_singleton_columns(SingletonTest& t, Plan& plan, const WorkingLp& lp, const Stats& stats, const gpp_params& p,
                           const int32_t* gate) {
  const int m = lp.m(), n = lp.n();
  auto s = ctx().stream;
  const ScArgs g = singleton_args(t, plan, lp, stats, p);
  GPP_LAUNCH_BYTES(sc_candidates, double(n) * 11 + 16.0 * n, grid_stride_blocks((int64_t(n) + 3) / 4), kThreads, 0, s, g,
                   gate);
  // Activity cache of the claimed rows, proposals and their staging follow with
  // no wait between: the kernels read the candidate and row counts on the
  // device, and the one answer, after the staging, tells what the rule did.
  if (plan.bounds_mirrored) GPP_LAUNCH(sc_cache<true>, g.row_blocks + g.long_blocks, kThreads, 0, s, g);
  else GPP_LAUNCH(sc_cache<false>, g.row_blocks + g.long_blocks, kThreads, 0, s, g);
  GPP_LAUNCH(sc_propose, grid_stride_blocks(n), kThreads, 0, s, g);
  t.report = ctx().open_report(kStWords, g.st);
  GPP_LAUNCH(sc_stage, grid_stride_blocks(std::min(m, n)), kThreads, 0, s, g, t.report);
  t.asked = true;
}

uint32_t probe_and_ask_singleton_columns(const ProbeArgs& probe, SingletonTest& t, Plan& plan, const WorkingLp& lp,
                                         const Stats& stats, const gpp_params& p) {
  auto s = ctx().stream;
  const ScArgs g = singleton_args(t, plan, lp, stats, p);
  const Report report = ctx().open_report(kStWords + 1, g.st);
  if (plan.bounds_mirrored)
    GPP_LAUNCH(probe_and_singleton_columns<true>, kSmallCluster, kThreads, 0, s, probe, g, report);
  else
    GPP_LAUNCH(probe_and_singleton_columns<false>, kSmallCluster, kThreads, 0, s, probe, g, report);
  const int64_t* f = ctx().await(report);
  std::copy(f, f + kStWords, t.answer);
  t.asked = t.answered = true;
  return uint32_t(f[kStWords]);
}

void rule_singleton_columns(Plan& plan, const WorkingLp& lp, const Stats& stats, const gpp_params& p,
                            SingletonTest* ahead) {
  if (plan.has_infeasible || plan.has_unbounded || !p.enable_singleton_columns) return;
  const int m = lp.m(), n = lp.n();
  if (m == 0 || n == 0) return;
  auto s = ctx().stream;
  SingletonTest own;
  SingletonTest& t = ahead && ahead->asked ? *ahead : own;
  if (!t.asked) {
    if (!plan.sc_ready) {
      if (plan.sc_owner.n < size_t(m)) plan.sc_owner.alloc(size_t(m), s);
      if (!plan.sc_words.p) plan.sc_words.alloc(kSingletonWords + 1, s);
      GPP_LAUNCH(sc_start, grid_stride_blocks(m), kThreads, 0, s, plan.sc_owner.p, m, kUnclaimed, plan.sc_words.p);
    }
    ask_singleton_columns(t, plan, lp, stats, p, nullptr);
  }
  plan.sc_ready = false;
  DBuf<int32_t>& owner = plan.sc_owner;
  int32_t* const st = plan.sc_words.p;
  const int claims = std::min(m, n);
  DBuf<int32_t>& winners = t.winners;
  DBuf<uint8_t>& kind = t.kind;
  DBuf<int64_t>& contrib_idx = t.contrib_idx;
  DBuf<double>&contrib_val = t.contrib_val, &side = t.side;
  if (!t.answered) std::copy_n(ctx().await(t.report), int(kStWords), t.answer);
  const int64_t* f = t.answer;
  if (f[kStUnbounded]) { plan.has_unbounded = true; return; }
  const int nwin = int(f[kStWin]), nelim = int(f[kStElim]);
  const bool any_side = f[kStSide] != 0;
  if (nelim == 0 && !any_side) return;

  // Cost update of the columns sharing an eliminated row.
  if (nelim) {
    DBuf<uint32_t> claimed(size_t(n + 31) / 32, s);
    claimed.zero();
    DBuf<int32_t> touched(size_t(n), s);
    GPP_LAUNCH(sc_touch, std::max(1, std::min((nwin + 7) / 8, kNumSMs * 16)), kThreads, 0, s, winners.p, st,
               kind.p, lp.A.ptr, lp.A.idx, plan.keep_col.p, claimed.p, touched.p, st);
    GPP_LAUNCH(sc_cost, std::max(1, std::min((n + 7) / 8, kNumSMs * 16)), kThreads, 0, s, touched.p, st, n, lp.AT.ptr,
               lp.AT.idx, lp.AT.val, owner.p, stats.scol_val.p, plan.c.p);
  }

  // Records, in ascending row order: substitutions, then dual shifts.
  if (p.record_postsolve_tape && nwin) {
    DBuf<uint64_t> keys(size_t(nwin), s);
    DBuf<int32_t> sorted(size_t(nwin), s);
    GPP_LAUNCH(sc_winner_keys, grid_stride_blocks(nwin), kThreads, 0, s, winners.p, nwin, kind.p, keys.p, sorted.p);
    radix_sort_pairs(keys.p, sorted.p, nwin, s, (uint64_t(1) << 32) | bits_up_to(m - 1));
    const int nshift = nwin - nelim;
    if (nelim) {
      DBuf<int32_t> sel(size_t(nelim) + 1, s), rec(size_t(nelim) + 1, s);
      DBuf<int64_t> sup(size_t(nelim) + 1, s), spos(size_t(nelim) + 1, s);
      const int blocks = std::max(1, std::min((nelim + 7) / 8, kNumSMs * 16));
      GPP_LAUNCH(sc_sub_sizes, blocks, kThreads, 0, s, sorted.p, nelim, owner.p, lp.A.ptr, lp.A.idx, lp.A.val,
                 plan.keep_col.p, p.zero_tol, sel.p, sup.p);
      const uint32_t seq = ctx().open_mail();
      scan_items<int64_t, 2>(
          nelim,
          [sel = sel.p, sup = sup.p] __device__(int64_t i, int64_t(&v)[2]) {
            v[0] = sel[i];
            v[1] = sup[i];
          },
          [rec = rec.p, spos = spos.p] __device__(int64_t i, const int64_t(&before)[2], const int64_t(&)[2]) {
            rec[i] = int32_t(before[0]);
            spos[i] = before[1];
          },
          [rec = rec.p + nelim, spos = spos.p + nelim, mail = ctx().box(seq), seq] __device__(const int64_t(&sum)[2]) {
            *rec = int32_t(sum[0]);
            *spos = sum[1];
            post_values(mail, seq, sum[0], sum[1]);
          },
          s);
      const int64_t* sums = ctx().await(ctx().box(seq), seq, "substitution records");
      const int64_t recs = sums[0], support = sums[1];
      if (recs) {
        PostsolveSegment seg = make_segment(recs, 3 * recs + support, 6 * recs + support);
        GPP_LAUNCH(sc_sub_pack, blocks, kThreads, 0, s, sorted.p, nelim, owner.p, kind.p, sel.p, rec.p, spos.p,
                   lp.A.ptr, lp.A.idx, lp.A.val, plan.keep_col.p, side.p, plan.c.p, plan.l.p, plan.u.p,
                   seg.types.p, seg.is.p, seg.vs.p, seg.idx.p, seg.val.p);
        plan.tape.push_back(std::move(seg));
      }
    }
    if (nshift) {
      PostsolveSegment seg = make_segment(nshift, nshift, nshift);
      GPP_LAUNCH(sc_shift_pack, grid_stride_blocks(nshift), kThreads, 0, s, sorted.p + nelim, nshift, seg.types.p,
                 seg.is.p, seg.vs.p, seg.idx.p, seg.val.p);
      plan.tape.push_back(std::move(seg));
    }
  }

  if (nelim) {
    DBuf<double> contrib(size_t(n), s);
    contrib.zero();
    GPP_LAUNCH(sc_scatter_contrib, grid_stride_blocks(nelim), kThreads, 0, s, nelim, contrib_idx.p, contrib_val.p,
               contrib.p);
    plan.obj_delta += det_sum_later(contrib.p, nullptr, n, s);
  }
  plan.has_row_action = true;
  plan.has_col_action = plan.has_col_action || nelim > 0;
  plan.has_change = true;
}

}  // namespace gpp

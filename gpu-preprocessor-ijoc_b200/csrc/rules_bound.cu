// Bound strengthening: one Jacobi round of activity-based implied column
// bounds, finalisation (margins, near-fixing, free-zero-cost guard), support
// rows for the postsolve tape, and the fixed-column row shift.
//
// Reference: rules/rule_bound_strengthening.cu:336-813 (kernels) and
// :1176-1557 (driver).  Candidate bounds are combined with CAS max/min, whose
// result does not depend on the order of the updates.
#include <climits>

#include "engine.cuh"
#include "scan.cuh"

namespace gpp {

namespace {


// Implied bounds of the column of entry a from its row (reference :349-430).
__device__ __forceinline__ void implied_bounds(double a, double lj, double uj, double al, double au, double mn,
                                               double mx, int ni, int pi, double& il, double& iu) {
  double tmin, tmax;
  if (a >= 0.0) { tmin = a * lj; tmax = a * uj; } else { tmin = a * uj; tmax = a * lj; }
  double rmin, rmax;
  if (isfinite(tmin)) rmin = ni == 0 ? mn - tmin : -INFINITY;
  else if (tmin < 0.0) rmin = ni > 1 ? -INFINITY : mn;
  else rmin = mn;
  if (isfinite(tmax)) rmax = pi == 0 ? mx - tmax : INFINITY;
  else if (tmax > 0.0) rmax = pi > 1 ? INFINITY : mx;
  else rmax = mx;
  il = -INFINITY;
  iu = INFINITY;
  if (a > 0.0) {
    if (isfinite(al) && isfinite(rmax)) il = (al - rmax) / a;
    if (isfinite(au) && isfinite(rmin)) iu = (au - rmin) / a;
  } else {
    if (isfinite(au) && isfinite(rmin)) il = (au - rmin) / a;
    if (isfinite(al) && isfinite(rmax)) iu = (al - rmax) / a;
  }
}

struct CandArgs {
  const offset_t* ptr;
  const int32_t* idx;
  const double* val;
  const double2* lu;   // packed column bounds, removed columns marked
  RowRecords rows;
  double zero_tol;
  double* cand_l;
  double* cand_u;
};

// The row's sides and activity summary, loaded once per row.
struct RowCtx {
  double al, au, mn, mx;
  int ni, pi;
  bool live;
};
__device__ __forceinline__ RowCtx row_ctx(const RowRecords& rows, int i) {
  const uint8_t f = rows.flags[i];
  const double2 sides = rows.sums[2 * int64_t(i)], sums = rows.sums[2 * int64_t(i) + 1];
  return RowCtx{sides.x, sides.y, sums.x, sums.y, f & 3, f >> 2 & 3, (f & kRowLive) != 0};
}

// Candidate bounds of column j from one entry a of a row (reference
// :373-430); b holds the column's current bounds.
__device__ __forceinline__ void candidate_update(const CandArgs& g, const RowCtx& rc, int j, double a, double2 b) {
  const double ol = b.x, ou = b.y;
  double il, iu;
  implied_bounds(a, ol, ou, rc.al, rc.au, rc.mn, rc.mx, rc.ni, rc.pi, il, iu);
  double nl = ol, nu = ou;
  if (isfinite(il)) nl = fmax(nl, il);
  if (isfinite(iu)) nu = fmin(nu, iu);
  if (nl > ol) red_max_f64(&g.cand_l[j], nl);
  if (nu < ou) red_min_f64(&g.cand_u[j], nu);
}

// Entry-parallel form of the candidate sweep: the candidates are combined by
// atomic max / min, which is order-free, so instead of row roles every thread
// takes consecutive stored entries (coalesced loads, full memory-level
// parallelism) and finds their row by a binary search over the tile's row
// pointers, staged in shared memory.
constexpr int kTileRows = 2048;

__global__ void __launch_bounds__(kThreads)
candidates_entries(offset_t nnz, const int2* __restrict__ tile_rows, int parts, CandArgs g) {
  after_previous_kernel();
  __shared__ offset_t sptr[kTileRows + 1];
  const L2Hints hint = l2_hints();
  // A block takes a tile, or on small models one of its `parts` equal parts.
  const int part_entries = kEntryTile / parts;
  const int64_t tiles = (int64_t(nnz) + kEntryTile - 1) / kEntryTile;
  for (int64_t w = blockIdx.x; w < tiles * parts; w += gridDim.x) {
    if (w * part_entries >= nnz) break;   // block-uniform
    const offset_t base = offset_t(w * part_entries);
    const offset_t last = offset_t(min(int64_t(nnz), w * part_entries + part_entries) - 1);
    const int2 span = tile_rows[w / parts];   // rows of the tile's first and last entry
    const int r0 = span.x, r1 = span.y;
    const bool staged = r1 - r0 + 1 <= kTileRows;
    if (staged)
      for (int k = threadIdx.x; k <= r1 - r0 + 1; k += kThreads) sptr[k] = g.ptr[r0 + k];
    __syncthreads();
    // The next entry's index and value are loaded one iteration ahead, so an
    // entry's critical path starts at its gather.
    const int K = part_entries / kThreads;
    offset_t p = base + threadIdx.x;
    int j = p <= last ? ld_stream(g.idx + p, hint.stream) : -1;
    double a = p <= last ? ld_stream(g.val + p, hint.stream) : 0.0;
    for (int k = 0; k < K && p <= last; ++k, p += kThreads) {
      const offset_t pn = p + kThreads;
      const bool next = k + 1 < K && pn <= last;
      const int jn = next ? ld_stream(g.idx + pn, hint.stream) : -1;
      const double an = next ? ld_stream(g.val + pn, hint.stream) : 0.0;
      const int i = staged ? r0 + row_of(sptr, 0, r1 - r0 + 1, p) : row_of(g.ptr, r0, r1 + 1, p);
      // Every load of the entry at once (the column's bounds do not depend on
      // the row; the row's record and flags are lines that the warp's
      // neighbouring entries share), so an entry waits for one memory round
      // trip instead of two.
      const double2 b = ld_keep(g.lu + j, hint.keep);
      const RowCtx rc = row_ctx(g.rows, i);
      if (rc.live && !removed_column(b) && !(fabs(a) <= g.zero_tol)) candidate_update(g, rc, j, a, b);
      j = jn;
      a = an;
    }
    __syncthreads();
  }
}

// One column's outcome.
struct ColumnBounds {
  double l, u, fixed_at;
  bool l_changed, u_changed, fixed, infeasible;
};

// _kernel_finalize_bound_strengthening (reference :646-796) for a kept column
// with bounds lj, uj and candidates cl, cu.
__device__ __forceinline__ ColumnBounds finalize_column(double lj, double uj, double cl, double cu, double cj, double vmax,
                                                        bool preserve_free_zero_cost, double zero_tol, double ft,
                                                        double upper_relax) {
  ColumnBounds r{lj, uj, 0.0, false, false, false, false};
  double el = lj, eu = uj;
  if (isfinite(cl)) el = fmax(el, cl);
  if (isfinite(cu)) eu = fmin(eu, cu);
  if (el > eu + ft) { r.infeasible = true; return r; }
  const bool was_free = !isfinite(lj) && !isfinite(uj);   // the bounds at the phase's start
  const bool box = isfinite(cl) && isfinite(cu);
  const bool zero_cost = fabs(cj) <= zero_tol;
  const bool nearly_fixed = box && (cu <= cl || (cu - cl) * vmax <= ft);
  if (preserve_free_zero_cost && was_free && box && zero_cost && !nearly_fixed) { cl = lj; cu = uj; }
  if (isfinite(cl) && cl > lj && isfinite(uj)) {
    if (cl >= uj + ft) { r.infeasible = true; return r; }
    if (cl >= uj || (uj - cl) * vmax <= ft) { r.fixed = true; r.fixed_at = uj; r.l = uj; r.u = uj; }
  }
  if (!r.fixed && isfinite(cl) && cl > lj) {
    const bool tighten = !isfinite(lj) || ((cl - lj > ft * 1.0e4) && (cl - lj > 1.0e-2 * fabs(lj)));
    if (tighten) {
      if (cl != nearbyint(cl)) cl -= 0.5 * ft * fabs(cl);
      r.l = cl;
      r.l_changed = true;
    }
  }
  if (!r.fixed && isfinite(cu) && cu < uj && isfinite(r.l)) {
    if (cu <= r.l - ft) { r.infeasible = true; return r; }
    if (cu <= r.l || (cu - r.l) * vmax <= ft) { r.fixed = true; r.fixed_at = r.l; r.u = r.l; }
  }
  if (!r.fixed && isfinite(cu) && cu < uj) {
    const bool tighten = !isfinite(uj) || ((uj - cu > ft * 1.0e4) && (uj - cu > 1.0e-2 * fabs(uj)));
    if (tighten) {
      if (cu != nearbyint(cu)) cu += upper_relax * ft * fabs(cu);
      r.u = cu;
      r.u_changed = true;
    }
  }
  if (r.fixed) r.l_changed = r.u_changed = false;
  return r;
}

struct SupportArgs {
  const offset_t* at_ptr;
  const int32_t* at_idx;
  const double* at_val;
  const uint8_t* keep_row;
  RowRecords rows;
  double zero_tol, tol, support_tol;
};
// The largest |a| of a column over its kept rows (reference :789-809), which the
// finalisation needs where a candidate would move a bound, for tests of the form
// d * max <= ft alone.  `d_min` is the least d: once an entry makes it too large, so is
// every test's product with the maximum (both round monotonely), and the walk ends
// there, most often at the first entries.
template <int kBatch>
__device__ __forceinline__ void max_of_entries(const SupportArgs& g, int64_t p, offset_t end, int step, double& v) {
  int row[kBatch];
  double a[kBatch];
#pragma unroll
  for (int k = 0; k < kBatch; ++k) {
    const bool in = end - p > k * step;
    row[k] = in ? g.at_idx[p + k * step] : -1;
    a[k] = in ? g.at_val[p + k * step] : 0.0;
  }
#pragma unroll
  for (int k = 0; k < kBatch; ++k)
    if (row[k] >= 0 && g.keep_row[row[k]]) v = fmax(v, fabs(a[k]));
}
__device__ __forceinline__ bool max_decides(double v, double d_min, double ft) { return d_min > 0.0 && d_min * v > ft; }
// A thread walks its own column (`wanted`), the warp takes columns of more than
// kWideColumn entries together, and one of more than kLongRow that its first
// kWideColumn entries do not decide is left to a block (`deferred`).  All lanes call it.
constexpr int kWideColumn = 64;
__device__ __forceinline__ double column_max(const SupportArgs& g, int j, bool wanted, double d_min, double ft,
                                             bool& deferred) {
  const offset_t first = wanted ? g.at_ptr[j] : 0, end = wanted ? g.at_ptr[j + 1] : 0;
  double v = 0.0;
  if (first < end) max_of_entries<2>(g, first, end, 1, v);
  const bool more = end - first > 2 && !max_decides(v, d_min, ft), is_long = end - first > kLongRow;
  const bool wide = more && !is_long && end - first > kWideColumn;
  if (more && !wide) {
    const offset_t stop = is_long ? first + kWideColumn : end;
    for (int64_t p = int64_t(first) + 2; p < stop && !max_decides(v, d_min, ft); p += 4) max_of_entries<4>(g, p, stop, 1, v);
  }
  deferred = more && is_long && !max_decides(v, d_min, ft);
  const int lane = threadIdx.x & 31;
  for (unsigned left = __ballot_sync(0xffffffffu, wide); left; left &= left - 1) {
    const int src = __ffs(left) - 1;
    const offset_t f = __shfl_sync(0xffffffffu, first, src), e = __shfl_sync(0xffffffffu, end, src);
    const double d = __shfl_sync(0xffffffffu, d_min, src);
    double m = 0.0;
    for (int64_t p = f; p < e; p += 4 * 32) {   // at most kLongRow entries
      max_of_entries<4>(g, p + lane, e, 32, m);
      if (__any_sync(0xffffffffu, max_decides(m, d, ft))) break;
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, off));
    if (lane == src) v = m;
  }
  return v;
}
// The same by a block, for one column.
__device__ __forceinline__ double column_max_block(const SupportArgs& g, int j, double d_min, double ft) {
  __shared__ double warp_max[kThreads / 32];
  const offset_t end = g.at_ptr[j + 1];
  double v = 0.0;
  for (int64_t p = g.at_ptr[j]; p < end; p += 4 * kThreads) {
    max_of_entries<4>(g, p + threadIdx.x, end, kThreads, v);
    if (__syncthreads_or(max_decides(v, d_min, ft))) break;
  }
#pragma unroll
  for (int off = 16; off; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
  if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = v;
  __syncthreads();
  v = warp_max[0];
#pragma unroll
  for (int w = 1; w < kThreads / 32; ++w) v = fmax(v, warp_max[w]);
  __syncthreads();   // the next column reuses them
  return v;
}
// Support rows of a changed column (reference :815-960): the smallest row that
// implies each new bound, INT_MAX when none does; among the entries of one of
// `lanes` threads.
__device__ __forceinline__ void support_rows(const SupportArgs& g, int j, double lj, double uj, const ColumnBounds& b,
                                             int lane, int lanes, int& sl, int& su) {
  sl = su = INT_MAX;
  const bool want_l = b.l_changed && b.l > lj + g.tol, want_u = b.u_changed && b.u < uj - g.tol;
  // Four entries per round with every load issued before the first use
  // (one memory round trip per four entries); the support row is the
  // smallest qualifying row, which does not depend on the visiting order.
  constexpr int kBatch = 4;
  const offset_t end = g.at_ptr[j + 1];
  for (int64_t p0 = int64_t(g.at_ptr[j]) + kBatch * lane; p0 < end && (want_l || want_u); p0 += kBatch * lanes) {
    int row[kBatch];
    double a[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      row[k] = p0 + k < end ? g.at_idx[p0 + k] : -1;
      a[k] = p0 + k < end ? g.at_val[p0 + k] : 0.0;
    }
    RowCtx rc[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) rc[k] = row_ctx(g.rows, row[k] >= 0 ? row[k] : 0);
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      if (row[k] < 0 || !rc[k].live || fabs(a[k]) <= g.zero_tol) continue;
      double il, iu;
      implied_bounds(a[k], lj, uj, rc[k].al, rc[k].au, rc[k].mn, rc[k].mx, rc[k].ni, rc[k].pi, il, iu);
      if (want_l && isfinite(il) && fabs(il - b.l) <= g.support_tol) sl = min(sl, row[k]);
      if (want_u && isfinite(iu) && fabs(iu - b.u) <= g.support_tol) su = min(su, row[k]);
    }
  }
}

// What the finalisation leaves per column.  `change` bits: 1 lower, 2 upper
// bound moved, 4 fixed (at its new lower bound); new bounds and support rows
// stand for the moved ones only.  `before`: per tile of kThreads columns the
// records (x) and their indices (y) of the columns before it, and the totals.
struct FinalBounds {
  double *l, *u;
  uint8_t* change;
  int32_t *sup_l, *sup_u;
  uint32_t* tile_counts;
  longlong2* before;   // four indices a column: past 2^31 from 537 million columns on
  int32_t* deferred;   // columns left to the second launch, as many as report word 5 says
};
// A column's records and their indices, 16 bits each.
__device__ __forceinline__ uint32_t bound_records(uint32_t change, int sup_l, int sup_u) {
  const uint32_t lc = change & 1u, uc = change >> 1 & 1u;
  const uint32_t recs = lc + uc;
  return recs | (recs + (lc && sup_l != INT_MAX ? 1u : 0u) + (uc && sup_u != INT_MAX ? 1u : 0u)) << 16;
}

// What both launches of the finalisation work on.
struct FinalArgs {
  int n, tiles;
  const uint8_t* keep_col;
  const double *l, *u, *c;
  double *cand_l, *cand_u;
  double2* lu;
  int preserve_free_zero_cost;
  double ft, upper_relax;
  bool records;
  SupportArgs support;
  FinalBounds out;
};
// A column's bounds and candidates, and what its tests ask of the maximum.
struct ColumnState {
  double l, u, cl, cu;
  __device__ __forceinline__ ColumnState(const FinalArgs& g, int j, bool kept)
      : l(kept ? g.l[j] : 0.0), u(kept ? g.u[j] : 0.0), cl(kept ? g.cand_l[j] : 0.0), cu(kept ? g.cand_u[j] : 0.0) {}
  __device__ __forceinline__ bool moves() const { return (isfinite(cl) && cl > l) || (isfinite(cu) && cu < u); }
  __device__ __forceinline__ double d_min() const { return fmin(fmin(u - cl, cu - l), cu - cl); }
};
__device__ __forceinline__ void smallest_of_block(int& a, int& b) {
  __shared__ int warp_least[2][kThreads / 32];
  a = __reduce_min_sync(0xffffffffu, a);
  b = __reduce_min_sync(0xffffffffu, b);
  if ((threadIdx.x & 31) == 0) {
    warp_least[0][threadIdx.x >> 5] = a;
    warp_least[1][threadIdx.x >> 5] = b;
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) {
    a = min(a, warp_least[0][w]);
    b = min(b, warp_least[1][w]);
  }
  __syncthreads();   // the next column reuses them
}
// A kept column's outcome: flags to `found`, its change bits and its records
// (bound_records).  By a thread, or by all of a block, whose first thread writes.
template <int kLanes>
__device__ __forceinline__ uint32_t settle_column(const FinalArgs& g, int j, const ColumnState& s, double vmax,
                                                  uint32_t& found, uint32_t& mine) {
  const int lane = kLanes == 1 ? 0 : threadIdx.x;
  ColumnBounds b = finalize_column(s.l, s.u, s.cl, s.cu, g.c[j], vmax, g.preserve_free_zero_cost != 0,
                                   g.support.zero_tol, g.ft, g.upper_relax);
  if (b.infeasible) {
    found |= 1u;
    b = ColumnBounds{s.l, s.u, 0.0, false, false, false, false};
  }
  const uint32_t change = (b.l_changed ? 1u : 0u) | (b.u_changed ? 2u : 0u) | (b.fixed ? 4u : 0u);
  if (change) found |= b.fixed ? 4u : 0u;
  if (change & 3u) {
    found |= 2u;
    if (g.records) {
      int sl, su;
      support_rows(g.support, j, s.l, s.u, b, lane, kLanes, sl, su);
      if constexpr (kLanes > 1) smallest_of_block(sl, su);
      mine = bound_records(change, sl, su);
      if (lane == 0) {
        g.out.sup_l[j] = sl;
        g.out.sup_u[j] = su;
      }
    }
  }
  if (lane != 0) return change;
  if (change) {
    g.out.l[j] = b.l;
    g.out.u[j] = b.u;
    const double removed = __longlong_as_double(static_cast<long long>(kRemovedColumnBits));
    g.lu[j] = b.fixed ? make_double2(removed, removed) : make_double2(b.l, b.u);
  }
  if (__double_as_longlong(s.cl) != __double_as_longlong(b.l)) g.cand_l[j] = b.l;
  if (__double_as_longlong(s.cu) != __double_as_longlong(b.u)) g.cand_u[j] = b.u;
  return change;
}

// The sums of the tiles' counts before each tile, and the totals, to the report.
// One block.
__device__ __forceinline__ void sum_tiles(int tiles, const FinalBounds& out, const Report& report) {
  constexpr int kEach = 4;
  __shared__ int2 warp_totals[kThreads / 32];   // of 1,024 tiles at a time
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  longlong2 total = make_longlong2(0, 0);
  for (int first = 0; first < tiles; first += kThreads * kEach) {
    uint32_t v[kEach];
    int2 own = make_int2(0, 0);
#pragma unroll
    for (int k = 0; k < kEach; ++k) {
      const int t = first + int(threadIdx.x) * kEach + k;
      v[k] = t < tiles ? __ldcg(out.tile_counts + t) : 0u;
      own.x += int(v[k] & 0xffffu);
      own.y += int(v[k] >> 16);
    }
    int2 upto = own;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, upto.x, off), y = __shfl_up_sync(0xffffffffu, upto.y, off);
      if (lane >= off) { upto.x += x; upto.y += y; }
    }
    if (lane == 31) warp_totals[warp] = upto;
    __syncthreads();
    longlong2 at = make_longlong2(total.x + upto.x - own.x, total.y + upto.y - own.y);
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
      const int2 s = warp_totals[w];
      if (w < warp) { at.x += s.x; at.y += s.y; }
      total.x += s.x;
      total.y += s.y;
    }
#pragma unroll
    for (int k = 0; k < kEach; ++k) {
      const int t = first + int(threadIdx.x) * kEach + k;
      if (t < tiles) out.before[t] = at;
      at.x += int(v[k] & 0xffffu);
      at.y += int(v[k] >> 16);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out.before[tiles] = total;
    report.words[1] = int32_t(total.x);
    report.words[2] = int32_t(total.x >> 32);
    report.words[3] = int32_t(total.y);
    report.words[4] = int32_t(total.y >> 32);
  }
  __syncthreads();
}

// Finalisation, support rows and the records' positions (:970-1008) in one
// pass over the columns: a tile's records are counted as it goes, and the last
// block to finish sums the tiles' counts (commit_bounds ranks within the tile).
// A column whose bounds stand costs its reads alone; the packed bounds and the
// candidates, which the next sweep starts from, are written where they differ.
// Bound by DRAM (42 bytes a column) where bounds stand, by the gathers of the
// moved columns' rows else: 376 us a sweep of the 29.8M-nnz LP's 5M columns, 446
// before the maximum's walk ended early.  A form that handed its tiles out in order
// and looked back for the records before them took 69 us against 45 at 500,001
// columns.  Report: word 0 flags (1 infeasible, 2 a bound moves, 4 a column is
// fixed), 1-2 records, 3-4 indices (low half first), 5 deferred columns.
__global__ void __launch_bounds__(kThreads, 3) finalize_kernel(FinalArgs g, Report report) {
  after_previous_kernel();
  __shared__ uint32_t warp_sums[2][kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t found = 0;
  int turn = 0;
  for (int t = blockIdx.x; t < g.tiles; t += gridDim.x, turn ^= 1) {
    const int64_t j64 = int64_t(t) * kThreads + threadIdx.x;
    const int j = int(j64);
    const bool kept = j64 < g.n && g.keep_col[j] != 0;
    const ColumnState s(g, j, kept);
    bool deferred;
    const double vmax = column_max(g.support, j, s.moves(), s.d_min(), g.ft, deferred);
    uint32_t mine = 0;
    if (deferred) g.out.deferred[atomicAdd(report.words + 5, 1)] = j;
    if (j64 < g.n) g.out.change[j] = uint8_t(kept && !deferred ? settle_column<1>(g, j, s, vmax, found, mine) : 0u);
    if (!g.records) continue;
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0) warp_sums[turn][warp] = mine;
    __syncthreads();   // the other turn's sums are read before the next one
    if (threadIdx.x == 0) {
      uint32_t sum = 0;
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w) sum += warp_sums[turn][w];
      g.out.tile_counts[t] = sum;
    }
  }
  gather_flags(report, found);
  if (!last_to_report(report)) return;
  if (g.records) sum_tiles(g.tiles, g.out, report);
  post_words(report);
}
// The deferred columns, a block each, and the tiles' sums once more.  Seldom: most
// long columns are decided by their first entries.  300 columns of 10,000 entries
// whose bounds close took 8.9 ms in two sweeps of a form that gave them to warps, and 8
// of 150,000 entries 73 ms; with these launches 0.19 and 0.69 ms.
__global__ void __launch_bounds__(kThreads) finalize_deferred(FinalArgs g, int count, Report report) {
  after_previous_kernel();
  uint32_t found = 0;
  for (int q = blockIdx.x; q < count; q += gridDim.x) {
    const int j = g.out.deferred[q];
    const ColumnState s(g, j, true);
    const double vmax = column_max_block(g.support, j, s.d_min(), g.ft);
    uint32_t mine = 0;
    const uint32_t change = settle_column<kThreads>(g, j, s, vmax, found, mine);
    if (threadIdx.x == 0) {
      g.out.change[j] = uint8_t(change);
      if (mine) atomicAdd(g.out.tile_counts + j / kThreads, mine);
    }
  }
  gather_flags(report, found);
  if (!last_to_report(report)) return;
  if (g.records) sum_tiles(g.tiles, g.out, report);
  post_words(report);
}

constexpr int kVariableBoundChange = 11, kRowImpliedBoundChange = 12, kFixedVariable = 0;

// The bound records of a column (`records` set), then its new bounds and mask.
struct BoundRecords {
  int32_t* types;
  int64_t *is, *vs;
  int32_t* idx;
  double* val;
};
__global__ void __launch_bounds__(kThreads)
commit_bounds(int n, int tiles, FinalBounds f, bool records, BoundRecords rec, double* __restrict__ l,
              double* __restrict__ u, uint8_t* __restrict__ keep_col, uint8_t* __restrict__ fixed,
              double* __restrict__ fixed_at) {
  after_previous_kernel();
  __shared__ uint32_t warp_sums[2][kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int turn = 0;
  if (records && blockIdx.x == 0 && threadIdx.x == 0) { rec.is[0] = 0; rec.vs[0] = 0; }
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int64_t j64 = int64_t(t) * kThreads + threadIdx.x;
    const uint32_t change = j64 < n ? f.change[j64] : 0u;
    const int j = int(j64);
    if (fixed && j64 < n) {
      fixed[j] = (change & 4u) != 0;
      fixed_at[j] = (change & 4u) ? f.l[j] : 0.0;
    }
    const bool lc = change & 1u, uc = change & 2u;
    int sl = INT_MAX, su = INT_MAX;
    longlong2 at = make_longlong2(0, 0);
    if (records) {
      at = f.before[t];
      if (f.before[t + 1].x != at.x) {   // block-uniform: the tile has records
        if (lc || uc) { sl = f.sup_l[j]; su = f.sup_u[j]; }
        const uint32_t own = bound_records(change, sl, su);
        uint32_t upto = own;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const uint32_t v = __shfl_up_sync(0xffffffffu, upto, off);
          if (lane >= off) upto += v;
        }
        if (lane == 31) warp_sums[turn][warp] = upto;
        __syncthreads();   // the other turn's sums are read before the next one
        uint32_t rank = upto - own;
#pragma unroll
        for (int w = 0; w < kThreads / 32; ++w) rank += w < warp ? warp_sums[turn][w] : 0u;
        turn ^= 1;
        at.x += int(rank & 0xffffu);
        at.y += int(rank >> 16);
      }
    }
    if (!change) continue;
    const double nl = f.l[j], nu = f.u[j];
    if (records && (lc || uc)) {
      int64_t k = at.x, ip = at.y;
      double cur_l = l[j];
      const double cur_u = u[j];
      auto emit = [&](int sup, double a, double b, double c2, double d) {
        rec.types[k] = sup == INT_MAX ? kVariableBoundChange : kRowImpliedBoundChange;
        rec.idx[ip++] = j;
        if (sup != INT_MAX) rec.idx[ip++] = sup;
        rec.val[4 * k] = a; rec.val[4 * k + 1] = b; rec.val[4 * k + 2] = c2; rec.val[4 * k + 3] = d;
        rec.is[k + 1] = ip;
        rec.vs[k + 1] = 4 * (k + 1);
        ++k;
      };
      if (lc) {
        emit(sl, cur_l, cur_u, nl, cur_u);
        cur_l = nl;
      }
      if (uc) emit(su, cur_l, cur_u, cur_l, nu);
    }
    l[j] = nl;
    u[j] = nu;
    if (change & 4u) keep_col[j] = 0;
  }
}

// Row shift of the fixed columns, then removal of rows left without a live
// column (feasible sides) or the infeasibility flag (reference :1083-1156).
__global__ void shift_and_empty_rows(int m, const offset_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                                     const double* __restrict__ shift, const uint8_t* __restrict__ keep_col,
                                     uint8_t* __restrict__ keep_row, double* __restrict__ AL,
                                     double* __restrict__ AU, double ft, Report report) {
  after_previous_kernel();
  uint32_t infeasible = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    AL[i] -= shift[i];
    AU[i] -= shift[i];
    if (!keep_row[i]) continue;
    int cnt = 0;
    for (offset_t p = ptr[i]; p < ptr[i + 1] && cnt == 0; ++p) cnt += keep_col[idx[p]] != 0;
    if (cnt) continue;
    if (AL[i] <= ft && AU[i] >= -ft) keep_row[i] = 0;
    else infeasible = 1;
  }
  post_flags(report, infeasible);
}

// FixedVariable records of fixed columns: (col, kept rows...), (value, c, coefficients...).
__global__ void fixed_record_sizes(int n, const uint8_t* __restrict__ fx, const offset_t* __restrict__ at_ptr,
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
__global__ void fixed_record_pack(int n, const uint8_t* __restrict__ fx, const offset_t* __restrict__ at_ptr,
                                  const int32_t* __restrict__ at_idx, const double* __restrict__ at_val,
                                  const uint8_t* __restrict__ keep_row, const double* __restrict__ fixv,
                                  const double* __restrict__ c, const int64_t* __restrict__ rec_pos,
                                  const int64_t* __restrict__ nz_pos, int32_t* __restrict__ types,
                                  int64_t* __restrict__ is, int64_t* __restrict__ vs, int32_t* __restrict__ idx,
                                  double* __restrict__ val, double* __restrict__ obj_c, double* __restrict__ obj_v) {
  after_previous_kernel();
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    if (j == 0) { is[0] = 0; vs[0] = 0; }
    if (!fx[j]) continue;
    const int64_t k = rec_pos[j], base = nz_pos[j];
    int64_t ip = k + base, vp = 2 * k + base;
    types[k] = kFixedVariable;
    idx[ip++] = j;
    val[vp++] = fixv[j];
    val[vp++] = c[j];
    for (offset_t p = at_ptr[j]; p < at_ptr[j + 1]; ++p)
      if (keep_row[at_idx[p]]) { idx[ip++] = at_idx[p]; val[vp++] = at_val[p]; }
    is[k + 1] = ip;
    vs[k + 1] = vp;
    obj_c[k] = c[j];
    obj_v[k] = fixv[j];
  }
}

// Live rows binned by infinite-term count of their minimum and maximum
// activity (0, 1, 2, >= 3): the learned schedule's histogram features.
__global__ void inf_histogram(int m, const uint8_t* __restrict__ keep_row, const uint8_t* __restrict__ flags,
                              uint32_t* __restrict__ hist) {
  after_previous_kernel();
  __shared__ uint32_t bins[8];
  if (threadIdx.x < 8) bins[threadIdx.x] = 0;
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    if (!keep_row[i]) continue;
    atomicAdd(&bins[flags[i] & 3], 1u);
    atomicAdd(&bins[4 + (flags[i] >> 2 & 3)], 1u);
  }
  __syncthreads();
  if (threadIdx.x < 8 && bins[threadIdx.x]) atomicAdd(hist + threadIdx.x, bins[threadIdx.x]);
}

}  // namespace

void rule_bound_strengthening(Plan& plan, const WorkingLp& lp, const Stats& stats, const gpp_params& p) {
  if (plan.has_infeasible || plan.has_unbounded) return;
  const int m = lp.m(), n = lp.n();
  if (m == 0 || n == 0) return;
  auto s = ctx().stream;
  DBuf<double2> row_sums(2 * size_t(m), s);
  DBuf<uint8_t> row_flags(size_t(m), s);
  const RowRecords rows{row_sums.p, row_flags.p};
  // One packed bounds array serves the activity sweep, the candidate sweep
  // and the redundant-row test after them.
  mirror_bounds(plan, n, s);
  row_activity_records(lp.A, plan.lu.p, p.zero_tol, plan, stats.row_nnz.p, rows, s, stats.version);
  if (plan.inf_hist) {
    check(cudaMemsetAsync(plan.inf_hist, 0, 8 * sizeof(uint32_t), s), "inf_hist");
    GPP_LAUNCH(inf_histogram, grid_stride_blocks(m), kThreads, 0, s, m, plan.keep_row.p, row_flags.p,
               plan.inf_hist);
  }
  {
    CandArgs g{lp.A.ptr, lp.A.idx, lp.A.val, plan.lu.p, rows, p.zero_tol, plan.cand_l.p, plan.cand_u.p};
    const double bytes = 4.0 * (m + 1) + 12.0 * lp.A.nnz + 33.0 * m + 16.0 * n + 16.0 * n;
    const RowSchedule& sch = stored_schedule(lp.A);
    // Small models have fewer tiles than the GPU has room for blocks: parts of
    // tiles then, down to one entry a thread (18 us a sweep of a 10,000-entry
    // model with whole tiles, eight dependent rounds).
    int parts = 1;
    while (parts < kEntryTile / kThreads && sch.tiles * parts * 2 <= kNumSMs * 8) parts *= 2;
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>(sch.tiles * parts, kNumSMs * 8));
    GPP_LAUNCH_BYTES(candidates_entries, bytes, int(blocks), kThreads, 0, s, lp.A.nnz, sch.tile_rows.p, parts, g);
  }
  const bool records = p.record_postsolve_tape != 0;
  DBuf<double> fl(size_t(n), s), fu(size_t(n), s);
  DBuf<uint8_t> change(size_t(n), s);
  const int tiles = int((int64_t(n) + kThreads - 1) / kThreads);
  DBuf<int32_t> sl, su;
  DBuf<uint32_t> tile_counts;
  DBuf<longlong2> before;
  if (records) {
    sl.alloc(size_t(n), s);
    su.alloc(size_t(n), s);
    tile_counts.alloc(size_t(tiles), s);
    before.alloc(size_t(tiles) + 1, s);
  }
  DBuf<int32_t> deferred(size_t(n), s);
  const FinalBounds fin{fl.p, fu.p, change.p, sl.p, su.p, tile_counts.p, before.p, deferred.p};
  const double support_tol = std::fmax(10.0 * p.bound_tol, 1.0e-10);
  const SupportArgs support{lp.AT.ptr, lp.AT.idx, lp.AT.val, plan.keep_row.p, rows,
                            p.zero_tol, p.bound_tol, support_tol};
  const FinalArgs final_args{n, tiles, plan.keep_col.p, plan.l.p, plan.u.p, plan.c.p, plan.cand_l.p, plan.cand_u.p,
                             plan.lu.p, int(p.bound_strengthening_preserve_free_zero_cost), p.feasibility_tol,
                             p.bound_strengthening_upper_relaxation_factor, records, support, fin};
  Report report = ctx().open_report(6);
  GPP_LAUNCH(finalize_kernel, std::min(tiles, kNumSMs * 12), kThreads, 0, s, final_args, report);
  const int64_t* answer = ctx().await(report);
  uint32_t found = uint32_t(answer[0]);
  if (answer[5] && !(found & 1u)) {
    const int count = int(answer[5]);
    report = ctx().open_report(5);
    GPP_LAUNCH(finalize_deferred, std::min(count, kNumSMs * 8), kThreads, 0, s, final_args, count, report);
    answer = ctx().await(report);
    found |= uint32_t(answer[0]);
  }
  if (found & 1u) { plan.has_infeasible = true; return; }
  const bool changed = (found & 2u) != 0, fixed = (found & 4u) != 0;
  if (!changed && !fixed) return;
  BoundRecords rec{};
  PostsolveSegment seg;
  const auto count_of = [answer](int k) { return int64_t(uint32_t(answer[k])) | answer[k + 1] << 32; };
  const int64_t recs = count_of(1), nidx = count_of(3);
  if (recs) {
    seg = make_segment(recs, nidx, 4 * recs);
    rec = BoundRecords{seg.types.p, seg.is.p, seg.vs.p, seg.idx.p, seg.val.p};
  }
  DBuf<uint8_t> fx;
  DBuf<double> fixv;
  if (fixed) {
    if (plan.save_committed) plan.save_committed();
    fx.alloc(size_t(n), s);
    fixv.alloc(size_t(n), s);
  }
  GPP_LAUNCH(commit_bounds, std::min(tiles, kNumSMs * 8), kThreads, 0, s, n, tiles, fin, recs > 0, rec, plan.l.p, plan.u.p,
             plan.keep_col.p, fx.p, fixv.p);
  if (recs) plan.tape.push_back(std::move(seg));
  double obj_delta = 0.0;
  if (fixed) {
    DBuf<double> shift(size_t(m), s);
    row_gather_shift(lp.A, lp.AT, plan.keep_row.p, fx.p, fixv.p, nullptr, shift.p, s);
    report = ctx().open_report(1);
    GPP_LAUNCH(shift_and_empty_rows, grid_stride_blocks(m), kThreads, 0, s, m, lp.A.ptr, lp.A.idx, shift.p,
               plan.keep_col.p, plan.keep_row.p, plan.AL.p, plan.AU.p, p.feasibility_tol, report);
    if (ctx().await(report)[0]) { plan.has_infeasible = true; return; }
    DBuf<int64_t> rc(size_t(n) + 1, s), nz(size_t(n) + 1, s), rpos(size_t(n) + 1, s), npos(size_t(n) + 1, s);
    GPP_LAUNCH(fixed_record_sizes, grid_stride_blocks(n), kThreads, 0, s, n, fx.p, lp.AT.ptr, lp.AT.idx,
               plan.keep_row.p, rc.p, nz.p);
    const auto [recs, nnz] = exclusive_scan_pair_i64(rc.p, rpos.p, nz.p, npos.p, n, s);
    PostsolveSegment seg = make_segment(recs, recs + nnz, 2 * recs + nnz);
    DBuf<double> oc(size_t(recs), s), ov(size_t(recs), s);
    GPP_LAUNCH(fixed_record_pack, grid_stride_blocks(n), kThreads, 0, s, n, fx.p, lp.AT.ptr, lp.AT.idx, lp.AT.val,
               plan.keep_row.p, fixv.p, plan.c.p, rpos.p, npos.p, seg.types.p, seg.is.p, seg.vs.p, seg.idx.p,
               seg.val.p, oc.p, ov.p);
    // append_compact_fixed_variable_tape_from_device (fixed_variable_tape.cu:286-315):
    // objective delta accumulated in long double in column order.
    const auto [hc, hv] = to_host2(oc.p, size_t(recs), ov.p, size_t(recs));
    long double acc = 0.0L;
    for (size_t k = 0; k < hc.size(); ++k) acc += (long double)hc[k] * (long double)hv[k];
    obj_delta = double(acc);
    if (p.record_postsolve_tape) plan.tape.push_back(std::move(seg));
  }
  plan.obj_delta += obj_delta;
  plan.has_row_action = plan.has_row_action || fixed;
  plan.has_col_action = plan.has_col_action || fixed;
  plan.has_change = true;
}

}  // namespace gpp

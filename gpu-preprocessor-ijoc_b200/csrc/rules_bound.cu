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


struct RowSummary {
  const double* mn;
  const double* mx;
  const int32_t* ni;
  const int32_t* pi;
};

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
  const uint8_t* keep_row;
  const int32_t* row_nnz;
  const double* AL;
  const double* AU;
  const double2* lu;   // packed column bounds, removed columns marked
  RowSummary rs;
  double zero_tol;
  double* cand_l;
  double* cand_u;
};

// The row's sides and activity summary, loaded once per row.
struct RowCtx {
  double al, au, mn, mx;
  int ni, pi;
};
__device__ __forceinline__ RowCtx row_ctx(const CandArgs& g, int i) {
  return RowCtx{g.AL[i], g.AU[i], g.rs.mn[i], g.rs.mx[i], g.rs.ni[i], g.rs.pi[i]};
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
candidates_entries(offset_t nnz, const int2* __restrict__ tile_rows, CandArgs g) {
  __shared__ offset_t sptr[kTileRows + 1];
  const L2Hints hint = l2_hints();
  for (offset_t base = offset_t(blockIdx.x) * kEntryTile; base < nnz; base += offset_t(gridDim.x) * kEntryTile) {
    const offset_t last = min(nnz, base + kEntryTile) - 1;
    const int2 span = tile_rows[base / kEntryTile];   // rows of the tile's first and last entry
    const int r0 = span.x, r1 = span.y;
    const bool staged = r1 - r0 + 1 <= kTileRows;
    if (staged)
      for (int k = threadIdx.x; k <= r1 - r0 + 1; k += kThreads) sptr[k] = g.ptr[r0 + k];
    __syncthreads();
    // The next entry's index and value are loaded one iteration ahead, so an
    // entry's critical path starts at its gather.
    constexpr int K = kEntryTile / kThreads;
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
      // the row; the row's flags and summary come from one or two lines that
      // the warp's neighbouring entries share), so an entry waits for one
      // memory round trip instead of two.
      const double2 b = ld_keep(g.lu + j, hint.keep);
      const bool row_live = (g.keep_row[i] != 0) & (g.row_nnz[i] > 1);
      const RowCtx rc = row_ctx(g, i);
      if (row_live && !removed_column(b) && !(fabs(a) <= g.zero_tol)) candidate_update(g, rc, j, a, b);
      j = jn;
      a = an;
    }
    __syncthreads();
  }
}

// _kernel_finalize_bound_strengthening (reference :646-796).
__global__ void finalize_kernel(int n, const uint8_t* __restrict__ keep_col, const double* __restrict__ l,
                                const double* __restrict__ u, const double* __restrict__ cand_l,
                                const double* __restrict__ cand_u, const double* __restrict__ c,
                                const double* __restrict__ vmax_arr, int preserve_free_zero_cost, double zero_tol,
                                double ft, double upper_relax, double* __restrict__ fl, double* __restrict__ fu,
                                uint8_t* __restrict__ lch, uint8_t* __restrict__ uch, uint8_t* __restrict__ fx,
                                double* __restrict__ fixv, Report report, bool post) {
  uint32_t found = 0;   // 1 infeasible, 2 a bound moves, 4 a column is fixed
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const double lj = l[j], uj = u[j];
    if (!keep_col[j]) {
      fl[j] = lj; fu[j] = uj; lch[j] = uch[j] = fx[j] = 0; fixv[j] = 0.0;
      continue;
    }
    double cl = cand_l[j], cu = cand_u[j];
    const double vmax = vmax_arr[j];
    double nl = lj, nu = uj;
    uint8_t lc = 0, uc = 0, fj = 0;
    double fat = 0.0;
    double el = lj, eu = uj;
    if (isfinite(cl)) el = fmax(el, cl);
    if (isfinite(cu)) eu = fmin(eu, cu);
    if (el > eu + ft) { found |= 1u; lch[j] = uch[j] = 0; continue; }
    const bool was_free = !isfinite(lj) && !isfinite(uj);   // the bounds at the phase's start
    const bool box = isfinite(cl) && isfinite(cu);
    const bool zero_cost = fabs(c[j]) <= zero_tol;
    const bool nearly_fixed = box && (cu <= cl || (cu - cl) * vmax <= ft);
    if (preserve_free_zero_cost && was_free && box && zero_cost && !nearly_fixed) { cl = lj; cu = uj; }
    if (isfinite(cl) && cl > lj && isfinite(uj)) {
      if (cl >= uj + ft) { found |= 1u; lch[j] = uch[j] = 0; continue; }
      if (cl >= uj || (uj - cl) * vmax <= ft) { fj = 1; fat = uj; nl = uj; nu = uj; }
    }
    if (!fj && isfinite(cl) && cl > lj) {
      const bool tighten = !isfinite(lj) || ((cl - lj > ft * 1.0e4) && (cl - lj > 1.0e-2 * fabs(lj)));
      if (tighten) {
        if (cl != nearbyint(cl)) cl -= 0.5 * ft * fabs(cl);
        nl = cl;
        lc = 1;
      }
    }
    if (!fj && isfinite(cu) && cu < uj && isfinite(nl)) {
      if (cu <= nl - ft) { found |= 1u; lch[j] = uch[j] = 0; continue; }
      if (cu <= nl || (cu - nl) * vmax <= ft) { fj = 1; fat = nl; nu = nl; }
    }
    if (!fj && isfinite(cu) && cu < uj) {
      const bool tighten = !isfinite(uj) || ((uj - cu > ft * 1.0e4) && (uj - cu > 1.0e-2 * fabs(uj)));
      if (tighten) {
        if (cu != nearbyint(cu)) cu += upper_relax * ft * fabs(cu);
        nu = cu;
        uc = 1;
      }
    }
    if (fj) { lc = uc = 0; found |= 4u; }
    if (lc || uc) found |= 2u;
    fl[j] = nl; fu[j] = nu; lch[j] = lc; uch[j] = uc; fx[j] = fj; fixv[j] = fat;
  }
  if (post) post_flags(report, found);
  else gather_flags(report, found);
}

// Support rows (reference :815-960); the per-column tape sizes (:970-1008)
// follow from them in the scan.
__global__ void support_kernel(int n, const offset_t* __restrict__ at_ptr, const int32_t* __restrict__ at_idx,
                               const double* __restrict__ at_val, const uint8_t* __restrict__ keep_row,
                               const int32_t* __restrict__ row_nnz, const double* __restrict__ AL,
                               const double* __restrict__ AU, const double* __restrict__ l,
                               const double* __restrict__ u, RowSummary rs, const uint8_t* __restrict__ lch,
                               const uint8_t* __restrict__ uch, const double* __restrict__ fl,
                               const double* __restrict__ fu, double zero_tol, double tol, double support_tol,
                               int32_t* __restrict__ sup_l, int32_t* __restrict__ sup_u) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    int sl = INT_MAX, su = INT_MAX;
    const bool nl = lch[j], nu = uch[j];
    if (nl || nu) {
      const double lj = l[j], uj = u[j], flj = fl[j], fuj = fu[j];
      const bool want_l = nl && flj > lj + tol, want_u = nu && fuj < uj - tol;
      // Four entries per round with every load issued before the first use
      // (one memory round trip per four entries); the support row is the
      // smallest qualifying row, which does not depend on the visiting order.
      constexpr int kBatch = 4;
      const offset_t end = at_ptr[j + 1];
      for (offset_t p0 = at_ptr[j]; p0 < end && (want_l || want_u); p0 += kBatch) {
        int row[kBatch];
        double a[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          row[k] = p0 + k < end ? at_idx[p0 + k] : -1;
          a[k] = p0 + k < end ? at_val[p0 + k] : 0.0;
        }
        bool live[kBatch];
        double al[kBatch], au[kBatch], mn[kBatch], mx[kBatch];
        int ni[kBatch], pi[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          const int i = row[k] >= 0 ? row[k] : 0;
          live[k] = row[k] >= 0 && (keep_row[i] != 0) & (row_nnz[i] > 1);
          al[k] = AL[i]; au[k] = AU[i]; mn[k] = rs.mn[i]; mx[k] = rs.mx[i]; ni[k] = rs.ni[i]; pi[k] = rs.pi[i];
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          if (!live[k] || fabs(a[k]) <= zero_tol) continue;
          double il, iu;
          implied_bounds(a[k], lj, uj, al[k], au[k], mn[k], mx[k], ni[k], pi[k], il, iu);
          if (want_l && isfinite(il) && fabs(il - flj) <= support_tol) sl = min(sl, row[k]);
          if (want_u && isfinite(iu) && fabs(iu - fuj) <= support_tol) su = min(su, row[k]);
        }
      }
    }
    sup_l[j] = sl;
    sup_u[j] = su;
  }
}

constexpr int kVariableBoundChange = 11, kRowImpliedBoundChange = 12, kFixedVariable = 0;

// The bound records of a column (`records` set), then its new bounds and mask.
struct BoundRecords {
  const int32_t *sup_l, *sup_u, *rec_pos, *idx_pos;
  int32_t* types;
  int64_t *is, *vs;
  int32_t* idx;
  double* val;
};
__global__ void commit_bounds(int n, const uint8_t* __restrict__ lch, const uint8_t* __restrict__ uch,
                              const double* __restrict__ fl, const double* __restrict__ fu,
                              const uint8_t* __restrict__ fx, bool records, BoundRecords rec, double* __restrict__ l,
                              double* __restrict__ u, uint8_t* __restrict__ keep_col) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const double nl = fl[j], nu = fu[j];
    if (records) {
      if (j == 0) { rec.is[0] = 0; rec.vs[0] = 0; }
      const bool lc = lch[j], uc = uch[j];
      if (lc || uc) {
        int64_t k = rec.rec_pos[j], ip = rec.idx_pos[j];
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
          emit(rec.sup_l[j], cur_l, cur_u, nl, cur_u);
          cur_l = nl;
        }
        if (uc) emit(rec.sup_u[j], cur_l, cur_u, cur_l, nu);
      }
    }
    l[j] = nl;
    u[j] = nu;
    if (fx[j]) keep_col[j] = 0;
  }
}

// Row shift of the fixed columns, then removal of rows left without a live
// column (feasible sides) or the infeasibility flag (reference :1083-1156).
__global__ void shift_and_empty_rows(int m, const offset_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                                     const double* __restrict__ shift, const uint8_t* __restrict__ keep_col,
                                     uint8_t* __restrict__ keep_row, double* __restrict__ AL,
                                     double* __restrict__ AU, double ft, Report report) {
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
__global__ void inf_histogram(int m, const uint8_t* __restrict__ keep_row, const int32_t* __restrict__ ni,
                              const int32_t* __restrict__ pi, uint32_t* __restrict__ hist) {
  __shared__ uint32_t bins[8];
  if (threadIdx.x < 8) bins[threadIdx.x] = 0;
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    if (!keep_row[i]) continue;
    atomicAdd(&bins[min(ni[i], 3)], 1u);
    atomicAdd(&bins[4 + min(pi[i], 3)], 1u);
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
  DBuf<double> cl(size_t(n), s), cu(size_t(n), s), mn(size_t(m), s), mx(size_t(m), s), vmax(size_t(n), s);
  DBuf<int32_t> ni(size_t(m), s), pi(size_t(m), s);
  // One packed bounds array serves the activity sweep and the candidate sweep.
  DBuf<double2> lu(size_t(n), s);
  pack_bounds(plan.l.p, plan.u.p, plan.keep_col.p, n, lu.p, s, cl.p, cu.p);
  row_activity_summary_packed(lp.A, lu.p, p.zero_tol, plan.keep_row.p, stats.row_nnz.p, mn.p, mx.p, ni.p, pi.p, s,
                              stats.version);
  const RowSummary rs{mn.p, mx.p, ni.p, pi.p};
  if (plan.inf_hist) {
    check(cudaMemsetAsync(plan.inf_hist, 0, 8 * sizeof(uint32_t), s), "inf_hist");
    GPP_LAUNCH(inf_histogram, grid_stride_blocks(m), kThreads, 0, s, m, plan.keep_row.p, ni.p, pi.p, plan.inf_hist);
  }
  {
    CandArgs g{lp.A.ptr, lp.A.idx, lp.A.val, plan.keep_row.p, stats.row_nnz.p, plan.AL.p, plan.AU.p, lu.p, rs,
               p.zero_tol, cl.p, cu.p};
    const double bytes = 4.0 * (m + 1) + 12.0 * lp.A.nnz + double(m) + 4.0 * m + 16.0 * m + 24.0 * m + 16.0 * n +
                         16.0 * n;
    const RowSchedule& sch = stored_schedule(lp.A);
    GPP_LAUNCH_BYTES(candidates_entries, bytes, int(std::max<int64_t>(1, std::min<int64_t>(sch.tiles, kNumSMs * 8))),
                     kThreads, 0, s, lp.A.nnz, sch.tile_rows.p, g);
  }
  col_max_abs(lp.AT, plan.keep_row.p, vmax.p, s);
  DBuf<double> fl(size_t(n), s), fu(size_t(n), s), fixv(size_t(n), s);
  DBuf<uint8_t> lch(size_t(n), s), uch(size_t(n), s), fx(size_t(n), s);
  // Finalisation, support rows and the records' positions run in a row, with
  // one answer: what was found and the tape sizes.
  const bool records = p.record_postsolve_tape != 0;
  Report report = ctx().open_report(1);
  GPP_LAUNCH(finalize_kernel, grid_stride_blocks(n), kThreads, 0, s, n, plan.keep_col.p, plan.l.p, plan.u.p, cl.p,
             cu.p, plan.c.p, vmax.p, int(p.bound_strengthening_preserve_free_zero_cost), p.zero_tol,
             p.feasibility_tol, p.bound_strengthening_upper_relaxation_factor, fl.p, fu.p, lch.p, uch.p, fx.p,
             fixv.p, report, !records);
  DBuf<int32_t> sl, su, rpos, ipos;
  if (records) {
    sl.alloc(size_t(n), s);
    su.alloc(size_t(n), s);
    rpos.alloc(size_t(n), s);
    ipos.alloc(size_t(n), s);
    const double support_tol = std::fmax(10.0 * p.bound_tol, 1.0e-10);
    GPP_LAUNCH(support_kernel, grid_stride_blocks(n), kThreads, 0, s, n, lp.AT.ptr, lp.AT.idx, lp.AT.val,
               plan.keep_row.p, stats.row_nnz.p, plan.AL.p, plan.AU.p, plan.l.p, plan.u.p, rs, lch.p, uch.p, fl.p,
               fu.p, p.zero_tol, p.bound_tol, support_tol, sl.p, su.p);
    scan_items<int32_t, 2>(
        n,
        [lch = lch.p, uch = uch.p, sl = sl.p, su = su.p] __device__(int64_t j, int32_t(&v)[2]) {
          const bool nl = lch[j], nu = uch[j];
          v[0] = int(nl) + int(nu);
          if (v[0]) v[1] = (nl ? (sl[j] == INT_MAX ? 1 : 2) : 0) + (nu ? (su[j] == INT_MAX ? 1 : 2) : 0);
        },
        [rpos = rpos.p, ipos = ipos.p] __device__(int64_t j, const int32_t(&before)[2], const int32_t(&v)[2]) {
          if (!v[0]) return;
          rpos[j] = before[0];
          ipos[j] = before[1];
        },
        [report] __device__(const int32_t(&sum)[2]) {
          report.mail->words[1] = sum[0];
          report.mail->words[2] = sum[1];
          report.mail->words[0] = __ldcg(report.words);
          report.words[0] = 0;
          __threadfence_system();
          report.mail->seq = report.seq;
        },
        s);
  }
  const volatile int64_t* answer = ctx().await(report);
  const uint32_t found = uint32_t(answer[0]);
  if (found & 1u) { plan.has_infeasible = true; return; }
  const bool changed = (found & 2u) != 0, fixed = (found & 4u) != 0;
  if (!changed && !fixed) return;
  BoundRecords rec{};
  PostsolveSegment seg;
  const int64_t recs = records ? answer[1] : 0, nidx = records ? answer[2] : 0;
  if (recs) {
    seg = make_segment(recs, nidx, 4 * recs);
    rec = BoundRecords{sl.p, su.p, rpos.p, ipos.p, seg.types.p, seg.is.p, seg.vs.p, seg.idx.p, seg.val.p};
  }
  GPP_LAUNCH(commit_bounds, grid_stride_blocks(n), kThreads, 0, s, n, lch.p, uch.p, fl.p, fu.p, fx.p, recs > 0, rec,
             plan.l.p, plan.u.p, plan.keep_col.p);
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

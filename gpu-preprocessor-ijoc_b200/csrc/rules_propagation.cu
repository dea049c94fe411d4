// Propagation rules besides bound strengthening: infeasible / redundant rows
// and lock-based dual fixing.
//
// Reference: rules/rule_infeasible_and_redundant_rows.cu:46-331 and
// rules/rule_dual_fix.cu:203-645 (with the device-resident infinite-bound
// record layout of device_recovery.cu:350-412).
#include "engine.cuh"

namespace gpp {

namespace {

__global__ void redundant_apply(int m, const uint8_t* __restrict__ action, uint8_t* __restrict__ keep_row,
                                double* __restrict__ AL, double* __restrict__ AU) {
  after_previous_kernel();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    const uint8_t a = action[i];
    if (a == 1) keep_row[i] = 0;
    else if (a == 2) AL[i] = -INFINITY;
    else if (a == 3) AU[i] = INFINITY;
  }
}

// _kernel_dual_fix_candidates (rule_dual_fix.cu:205-309).
// Bound by the chain from a column's pointers over its entries to their rows,
// so four entries are loaded at once and a row answers with one byte (its mask
// and the finiteness of its sides, 17 bytes in three places otherwise).
__global__ void row_kinds_kernel(int m, const uint8_t* __restrict__ keep_row, const double* __restrict__ AL,
                                 const double* __restrict__ AU, uint8_t* __restrict__ kinds) {
  after_previous_kernel();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x)
    kinds[i] = row_kind(keep_row[i], AL[i], AU[i]);
}
__global__ void dual_fix_candidates(int n, const uint8_t* __restrict__ keep_col, const uint8_t* __restrict__ kinds,
                                    const double* __restrict__ c, const double* __restrict__ l,
                                    const double* __restrict__ u, const offset_t* __restrict__ at_ptr,
                                    const int32_t* __restrict__ at_idx, const double* __restrict__ at_val,
                                    double zt, double bound_tol, int max_degree, const int32_t* __restrict__ col_nnz,
                                    uint8_t* __restrict__ fixed, uint8_t* __restrict__ inf_fix,
                                    double* __restrict__ fval, double* __restrict__ contrib, Report report) {
  after_previous_kernel();
  uint32_t found = 0;   // 1 infeasible, 2 unbounded, 4 a column is fixed, 8 at an infinite bound
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    fixed[j] = 0; inf_fix[j] = 0; fval[j] = 0.0; contrib[j] = 0.0;
    if (!keep_col[j]) continue;
    const double lj = l[j], uj = u[j];
    if (lj > uj + bound_tol) { found |= 1u; continue; }
    const double cj = c[j];
    if (fabs(cj) > zt && col_nnz[j] > max_degree) continue;
    bool down = false, up = false;
    const offset_t end = at_ptr[j + 1];
    for (offset_t p = at_ptr[j]; p < end && !(down && up); p += 4) {
      int row[4];
      double a[4];
      uint8_t kind[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        row[k] = p + k < end ? at_idx[p + k] : -1;
        a[k] = p + k < end ? at_val[p + k] : 0.0;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) kind[k] = row[k] >= 0 ? kinds[row[k]] : uint8_t(0);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint8_t low = a[k] > zt ? kRowLower : a[k] < -zt ? kRowUpper : uint8_t(0);
        if (low) {
          down = down || (kind[k] & low);
          up = up || (kind[k] & ((kRowLower | kRowUpper) ^ low));
        }
      }
    }
    bool f = false, fi = false;
    double v = 0.0;
    if (cj > zt) {
      if (!down) { if (isfinite(lj)) { v = lj; f = true; } else { found |= 2u; continue; } }
    } else if (cj < -zt) {
      if (!up) { if (isfinite(uj)) { v = uj; f = true; } else { found |= 2u; continue; } }
    } else if (fabs(cj) <= zt) {
      if (!down) { f = true; if (isfinite(lj)) v = lj; else { v = -INFINITY; fi = true; } }
      else if (!up) { f = true; if (isfinite(uj)) v = uj; else { v = INFINITY; fi = true; } }
    }
    if (f) {
      fixed[j] = 1; inf_fix[j] = fi; fval[j] = v; contrib[j] = fi ? 0.0 : cj * v;
      found |= fi ? 12u : 4u;
    }
  }
  post_flags(report, found);
}
__global__ void finite_fixed_mask(int n, const uint8_t* __restrict__ fixed, const uint8_t* __restrict__ inf_fix,
                                  uint8_t* __restrict__ out) {
  after_previous_kernel();
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
    out[j] = fixed[j] && !inf_fix[j];
}
__global__ void dual_fix_row_remove(int n, const uint8_t* __restrict__ fixed, const uint8_t* __restrict__ inf_fix,
                                    const uint8_t* __restrict__ keep_row, const offset_t* __restrict__ at_ptr,
                                    const int32_t* __restrict__ at_idx, uint8_t* __restrict__ remove,
                                    Report report) {
  after_previous_kernel();
  uint32_t any = 0;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    if (!(fixed[j] && inf_fix[j])) continue;
    for (offset_t p = at_ptr[j]; p < at_ptr[j + 1]; ++p)
      if (keep_row[at_idx[p]]) { remove[at_idx[p]] = 1; any = 1; }
  }
  post_flags(report, any);
}
// InfiniteBoundDualFix record sizes: 1 record per column, 3 + rows + entries
// indices and 1 + rows + entries values (entries restricted to the entry domain).
__global__ void infinite_sizes(int n, const uint8_t* __restrict__ fixed, const uint8_t* __restrict__ inf_fix,
                               const uint8_t* __restrict__ keep_row, const uint8_t* __restrict__ entry,
                               const offset_t* __restrict__ a_ptr, const int32_t* __restrict__ a_idx,
                               const offset_t* __restrict__ at_ptr, const int32_t* __restrict__ at_idx,
                               int64_t* __restrict__ recs, int64_t* __restrict__ sizes) {
  after_previous_kernel();
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const bool sel = fixed[j] && inf_fix[j];
    int64_t size = 0;
    if (sel)
      for (offset_t p = at_ptr[j]; p < at_ptr[j + 1]; ++p) {
        const int row = at_idx[p];
        if (!keep_row[row]) continue;
        ++size;
        for (offset_t q = a_ptr[row]; q < a_ptr[row + 1]; ++q) size += entry[a_idx[q]] != 0;
      }
    recs[j] = sel;
    sizes[j] = size;
  }
}
__global__ void infinite_pack(int n, const uint8_t* __restrict__ fixed, const uint8_t* __restrict__ inf_fix,
                              const double* __restrict__ fval, const uint8_t* __restrict__ keep_row,
                              const uint8_t* __restrict__ entry, const double* __restrict__ l,
                              const double* __restrict__ u, const double* __restrict__ AL,
                              const double* __restrict__ AU, const offset_t* __restrict__ a_ptr,
                              const int32_t* __restrict__ a_idx, const double* __restrict__ a_val,
                              const offset_t* __restrict__ at_ptr, const int32_t* __restrict__ at_idx,
                              const int64_t* __restrict__ rpos, const int64_t* __restrict__ spos,
                              int32_t* __restrict__ types, int64_t* __restrict__ is, int64_t* __restrict__ vs,
                              int32_t* __restrict__ idx, double* __restrict__ val) {
  after_previous_kernel();
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    if (j == 0) { is[0] = 0; vs[0] = 0; }
    if (!(fixed[j] && inf_fix[j])) continue;
    const int64_t k = rpos[j], base = spos[j];
    int64_t ip = base + 3 * k, vp = base + k;
    const bool pos = fval[j] > 0;
    types[k] = 1;  // InfiniteBoundDualFix
    idx[ip++] = pos ? 1 : -1;
    idx[ip++] = j;
    const int64_t count_pos = ip++;
    val[vp++] = pos ? l[j] : u[j];
    int active = 0;
    for (offset_t p = at_ptr[j]; p < at_ptr[j + 1]; ++p) {
      const int row = at_idx[p];
      if (!keep_row[row]) continue;
      ++active;
      const int64_t header = ip++;
      int len = 0;
      val[vp++] = isfinite(AL[row]) ? AL[row] : AU[row];
      for (offset_t q = a_ptr[row]; q < a_ptr[row + 1]; ++q) {
        if (!entry[a_idx[q]]) continue;
        ++len;
        idx[ip++] = a_idx[q];
        val[vp++] = a_val[q];
      }
      idx[header] = len;
    }
    idx[count_pos] = active;
    is[k + 1] = ip;
    vs[k + 1] = vp;
  }
}
__global__ void dual_fix_apply(int n, int m, const uint8_t* __restrict__ fixed, const double* __restrict__ fval,
                               const uint8_t* __restrict__ remove, const double* __restrict__ shift,
                               uint8_t* __restrict__ keep_col, uint8_t* __restrict__ keep_row,
                               double* __restrict__ l, double* __restrict__ u, double* __restrict__ AL,
                               double* __restrict__ AU) {
  after_previous_kernel();
  const int top = n > m ? n : m;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < top; k += gridDim.x * blockDim.x) {
    if (k < n && fixed[k]) { l[k] = fval[k]; u[k] = fval[k]; keep_col[k] = 0; }
    if (k < m) {
      AL[k] -= shift[k];
      AU[k] -= shift[k];
      if (remove && remove[k]) keep_row[k] = 0;
    }
  }
}

}  // namespace

void ask_dual_fix(DualFixTest& t, Plan& plan, const WorkingLp& lp, const Stats& stats, const gpp_params& p) {
  const int n = lp.n();
  auto s = ctx().stream;
  t.fixed.alloc(size_t(n), s);
  t.inf_fix.alloc(size_t(n), s);
  t.fval.alloc(size_t(n), s);
  t.contrib.alloc(size_t(n), s);
  t.report = ctx().open_report(1);
  GPP_LAUNCH(dual_fix_candidates, grid_stride_blocks(n), kThreads, 0, s, n, plan.keep_col.p, plan.row_kinds.p,
             plan.c.p, plan.l.p, plan.u.p, lp.AT.ptr, lp.AT.idx, lp.AT.val, p.zero_tol, p.bound_tol,
             p.dual_fix_max_nonzero_cost_col_degree, stats.col_nnz.p, t.fixed.p, t.inf_fix.p, t.fval.p, t.contrib.p,
             t.report);
  t.asked = true;
}

// `ahead`: dual fixing follows, and its test is launched before this rule's
// answer is waited for.  In a round without redundant rows, most of them, that
// takes one wait of about 8 us out; in the others a sweep over the columns is
// wasted, so up to kAskAhead entries only (a sweep takes 25 us there, 160 us on
// the 29.8M-nnz LP).
constexpr offset_t kAskAhead = 4 << 20;
void rule_redundant_rows(Plan& plan, const WorkingLp& lp, const Stats& stats, const gpp_params& p,
                         DualFixTest* ahead) {
  if (plan.has_infeasible || plan.has_unbounded) return;
  const int m = lp.m();
  if (m == 0) return;
  auto s = ctx().stream;
  DBuf<uint8_t> action(size_t(m), s);
  if (plan.row_kinds.n < size_t(m)) plan.row_kinds.alloc(size_t(m), s);
  plan.row_kinds_current = false;
  mirror_bounds(plan, lp.n(), s);
  const Report report = ctx().open_report(1);
  redundant_rows_test(lp.A, plan.lu.p, plan.keep_row.p, stats.row_nnz.p,
                      RedundantTest{plan.AL.p, plan.AU.p, p.bound_tol, action.p, plan.row_kinds.p, report}, s,
                      stats.version);
  if (ahead && lp.n() > 0 && lp.A.nnz <= kAskAhead) ask_dual_fix(*ahead, plan, lp, stats, p);
  const uint32_t found = uint32_t(ctx().await(report)[0]);
  if (found & 1u) { plan.has_infeasible = true; return; }
  if (!found) {
    plan.row_kinds_current = true;
    return;
  }
  const bool deleted = (found & 2u) != 0;
  GPP_LAUNCH(redundant_apply, grid_stride_blocks(m), kThreads, 0, s, m, action.p, plan.keep_row.p, plan.AL.p,
             plan.AU.p);
  plan.has_row_action = true;
  plan.has_redundant_row_deletion = plan.has_redundant_row_deletion || deleted;
  plan.has_row_deletion = plan.has_row_deletion || deleted;
  plan.has_change = true;
}

void rule_dual_fix(Plan& plan, const WorkingLp& lp, const Stats& stats, const gpp_params& p, DualFixTest* ahead) {
  if (plan.has_infeasible || plan.has_unbounded) return;
  const int n = lp.n(), m = lp.m();
  if (n == 0) return;
  auto s = ctx().stream;
  const bool stands = std::exchange(plan.row_kinds_current, false);   // no row acted on since
  DualFixTest own;
  DualFixTest& test = stands && ahead && ahead->asked ? *ahead : own;
  if (!test.asked) {
    if (!stands && m) {
      if (plan.row_kinds.n < size_t(m)) plan.row_kinds.alloc(size_t(m), s);
      GPP_LAUNCH(row_kinds_kernel, grid_stride_blocks(m), kThreads, 0, s, m, plan.keep_row.p, plan.AL.p, plan.AU.p,
                 plan.row_kinds.p);
    }
    ask_dual_fix(test, plan, lp, stats, p);
  }
  DBuf<uint8_t>&fixed = test.fixed, &inf_fix = test.inf_fix;
  DBuf<double>&fval = test.fval, &contrib = test.contrib;
  DBuf<uint8_t> finite, remove;
  DBuf<double> shift(size_t(std::max(m, 1)), s);
  Report report = test.report;
  const uint32_t found = uint32_t(ctx().await(report)[0]);
  if (found & 2u) { plan.has_unbounded = true; return; }
  if (found & 1u) { plan.has_infeasible = true; return; }
  if (!found) return;
  const bool any_inf = (found & 8u) != 0;
  // Columns fixed at an infinite bound shift no row and take their rows with
  // them; without any, every fixed column shifts its rows.
  if (any_inf) {
    finite.alloc(size_t(n), s);
    remove.alloc(size_t(std::max(m, 1)), s);
    GPP_LAUNCH(finite_fixed_mask, grid_stride_blocks(n), kThreads, 0, s, n, fixed.p, inf_fix.p, finite.p);
  }
  if (m) row_gather_shift(lp.A, lp.AT, plan.keep_row.p, any_inf ? finite.p : fixed.p, fval.p, nullptr, shift.p, s);
  bool row_changed = false;
  if (any_inf) {
    remove.zero();
    report = ctx().open_report(1);
    GPP_LAUNCH(dual_fix_row_remove, grid_stride_blocks(n), kThreads, 0, s, n, fixed.p, inf_fix.p, plan.keep_row.p,
               lp.AT.ptr, lp.AT.idx, remove.p, report);
    row_changed = ctx().await(report)[0] != 0;
  }
  if (p.record_postsolve_tape && any_inf) {
    DBuf<int64_t> rc(size_t(n) + 1, s), sz(size_t(n) + 1, s), rpos(size_t(n) + 1, s), spos(size_t(n) + 1, s);
    GPP_LAUNCH(infinite_sizes, grid_stride_blocks(n), kThreads, 0, s, n, fixed.p, inf_fix.p, plan.keep_row.p,
               plan.rule_entry_keep_col, lp.A.ptr, lp.A.idx, lp.AT.ptr, lp.AT.idx, rc.p, sz.p);
    const auto [recs, size] = exclusive_scan_pair_i64(rc.p, rpos.p, sz.p, spos.p, n, s);
    if (recs) {
      PostsolveSegment seg = make_segment(recs, size + 3 * recs, size + recs);
      GPP_LAUNCH(infinite_pack, grid_stride_blocks(n), kThreads, 0, s, n, fixed.p, inf_fix.p, fval.p, plan.keep_row.p,
                 plan.rule_entry_keep_col, plan.l.p, plan.u.p, plan.AL.p, plan.AU.p, lp.A.ptr, lp.A.idx, lp.A.val,
                 lp.AT.ptr, lp.AT.idx, rpos.p, spos.p, seg.types.p, seg.is.p, seg.vs.p, seg.idx.p, seg.val.p);
      plan.tape.push_back(std::move(seg));
    }
  }
  GPP_LAUNCH(dual_fix_apply, grid_stride_blocks(std::max(n, m)), kThreads, 0, s, n, m, fixed.p, fval.p, remove.p,
             shift.p, plan.keep_col.p, plan.keep_row.p, plan.l.p, plan.u.p, plan.AL.p, plan.AU.p);
  plan.obj_delta += domain_objective(contrib.p, plan.rule_entry_keep_col, n, s);
  plan.has_row_action = plan.has_row_action || row_changed;
  plan.has_col_action = plan.has_change = true;
}

}  // namespace gpp

// Postsolve: scatter the reduced solution to the original index space,
// restore fixed values, replay the tape in reverse (primal pass, then dual
// pass), and project reduced costs z = proj(c - A^T y) for the columns no
// record recovered exactly.
//
// Reference: postsolve_gpu (cpp/src/presolve/gpu_postsolve.cu:535-670) and the
// record handlers in cpp/src/presolve/postsolve/*.cuh.  The per-record
// arithmetic is the reference's; records that share a resource are replayed
// in reverse chronological order by one thread, independent groups of records
// in parallel, and the closing projection runs one thread per column.
#include "presolve.hpp"
#include "sort.hpp"

namespace gpp {

namespace {

constexpr double kTol = 1e-7;
enum : int {
  kFixedVariable = 0, kInfiniteBoundDualFix = 1, kSingletonColumnSubstitution = 2, kParallelColumn = 3,
  kParallelRow = 4, kDeletedRow = 5, kRowDualShift = 10, kRowImpliedBoundChange = 12, kDoubletonEquation = 13,
  kFmeCol = 14
};

__device__ __forceinline__ bool pfin(double x) { return x > -INFINITY && x < INFINITY; }
__device__ __forceinline__ bool at_lower(double x, double l, double tol) { return pfin(l) && x <= l + tol; }
__device__ __forceinline__ bool at_upper(double x, double u, double tol) { return pfin(u) && x >= u - tol; }
__device__ __forceinline__ double clamp_inf(double x, double lo, double hi) {
  double y = x;
  if (pfin(lo)) y = fmax(y, lo);
  if (pfin(hi)) y = fmin(y, hi);
  return y;
}

struct Model {
  const offset_t *A_ptr, *AT_ptr;
  const int32_t *A_idx, *AT_idx;
  const double *A_val, *AT_val, *c, *l, *u;
  bool present;
};
struct Sol {
  double *x, *y, *z;
  uint8_t* got;
};

__device__ double merged_source_value(double lo, double hi, double tol) {
  if (isfinite(lo) && isfinite(hi)) return 0.5 * (lo + hi);
  if (isfinite(lo)) { if (0.0 > lo + tol) return 0.0; return lo + fmax(1.0, fabs(lo) * fmax(tol, 1.0e-12)); }
  if (isfinite(hi)) { if (0.0 < hi - tol) return 0.0; return hi - fmax(1.0, fabs(hi) * fmax(tol, 1.0e-12)); }
  return 0.0;
}

__device__ void replay_record(int type, const int32_t* id, int64_t ni, const double* v, int64_t nv, Sol s,
                              const Model& M, bool primal, bool dual) {
  const double tol = kTol;
  double* x = s.x;
  double* y = s.y;
  double* z = s.z;
  if (type == kParallelColumn) {
    // replay_parallel_column (postsolve_parallel_columns.cuh:101-131).
    const int from = id[0], to = id[1];
    const double r = v[0], lo = v[1], hi = v[2], tl = v[3], tu = v[4];
    if (primal) {
      const double yv = x[to], zt = z ? z[to] : 0.0;
      double slo = lo, shi = hi;
      if (isfinite(tu)) { const double b = (yv - tu) / r; if (r > 0.0) slo = fmax(slo, b); else shi = fmin(shi, b); }
      if (isfinite(tl)) { const double b = (yv - tl) / r; if (r > 0.0) shi = fmin(shi, b); else slo = fmax(slo, b); }
      double lower = -INFINITY, upper = INFINITY;
      if (r > 0.0) { if (isfinite(tl) && isfinite(lo)) lower = tl + r * lo; }
      else if (isfinite(tl) && isfinite(hi)) lower = tl + r * hi;
      if (r > 0.0) { if (isfinite(tu) && isfinite(hi)) upper = tu + r * hi; }
      else if (isfinite(tu) && isfinite(lo)) upper = tu + r * lo;
      double xf;
      if (zt > tol && isfinite(lower) && fabs(yv - lower) <= tol) xf = r > 0.0 ? lo : hi;
      else if (zt < -tol && isfinite(upper) && fabs(yv - upper) <= tol) xf = r > 0.0 ? hi : lo;
      else xf = merged_source_value(slo, shi, tol);
      x[from] = xf;
      x[to] = yv - r * xf;
    }
    if (dual && z) { z[from] = r * z[to]; s.got[from] = 1; }
  } else if (type == kDoubletonEquation) {
    // replay_doubleton_equation (postsolve_doubleton_equations.cuh:88-172).
    const int ec = id[0], kc = id[1], row = id[2];
    const double ecoef = v[0], kcoef = v[1], rhs = v[2], eobj = v[9];
    const double alpha = -kcoef / ecoef, beta = rhs / ecoef;
    if (primal) x[ec] = beta + alpha * x[kc];
    if (dual && z && y && M.present) {
      const double okl = v[5], oku = v[6], nkl = v[7], nku = v[8];
      const double lsrc = nv >= 11 ? v[10] : 0.0, usrc = nv >= 12 ? v[11] : 0.0;
      double zk = 0.0, ze = 0.0;
      const double xk = x[kc], zkh = z[kc];
      if (fabs(alpha) <= tol) { zk = zkh; ze = 0.0; }
      else {
        const bool al = pfin(nkl) && xk <= nkl + tol, au = pfin(nku) && xk >= nku - tol;
        if (!al && !au) { zk = 0.0; ze = 0.0; }
        else {
          double src = al ? lsrc : usrc;
          if (src == 0.0) {
            if (al) src = (pfin(okl) && fabs(nkl - okl) <= tol) ? 1.0 : 2.0;
            else src = (pfin(oku) && fabs(nku - oku) <= tol) ? 1.0 : 2.0;
          }
          if (src == 2.0) { zk = 0.0; ze = zkh / alpha; } else { zk = zkh; ze = 0.0; }
        }
      }
      double sum_other = 0.0;
      if (ni >= 4 && nv >= 12) {
        const int cnt = id[3];
        for (int q = 0; q < cnt; ++q) sum_other += v[12 + q] * y[id[4 + q]];
        y[row] = (eobj - sum_other - ze) / ecoef;
      } else {
        for (offset_t q = M.AT_ptr[ec]; q < M.AT_ptr[ec + 1]; ++q)
          if (M.AT_idx[q] != row) sum_other += M.AT_val[q] * y[M.AT_idx[q]];
        y[row] = (M.c[ec] - sum_other - ze) / ecoef;
      }
      z[kc] = zk; z[ec] = ze; s.got[kc] = 1; s.got[ec] = 1;
    } else if (dual) {
      if (z) { z[ec] = 0.0; s.got[ec] = 1; }
      if (y && row >= 0) y[row] = eobj / ecoef;
    }
  } else if (type == kSingletonColumnSubstitution) {
    // replay_singleton_column_substitution (postsolve_singleton_columns.cuh:8-50).
    const int ec = id[0], row = id[1], cnt = id[2];
    const double piv = v[0], rhs = v[1], eobj = v[4];
    const bool deleted = v[5] != 0.0;
    double part = 0.0;
    for (int q = 0; q < cnt; ++q) part += v[6 + q] * x[id[3 + q]];
    if (primal) x[ec] = (rhs - part) / piv;
    if (dual && y && row >= 0) { if (deleted) y[row] = eobj / piv; else y[row] += eobj / piv; }
    if (dual && z) { z[ec] = deleted || !y ? 0.0 : eobj - piv * y[row]; s.got[ec] = 1; }
  } else if (type == kFixedVariable) {
    // replay_fixed_variable (postsolve_fixed_variables.cuh:8-40).
    const int col = id[0];
    if (primal) x[col] = v[0];
    if (dual && z) {
      double zj = v[1];
      if (y) for (int64_t q = 1; q < ni; ++q) zj -= v[2 + (q - 1)] * y[id[q]];
      z[col] = zj;
      s.got[col] = 1;
    }
  } else if (type == kInfiniteBoundDualFix) {
    // replay_infinite_bound_dual_fix (postsolve_fixed_variables.cuh:42-89).
    const bool pos = id[0] > 0;
    const int col = id[1], nrows = id[2];
    double ext = v[0];
    int64_t ip = 3, vp = 1;
    if (primal) {
      for (int r = 0; r < nrows; ++r) {
        const int len = id[ip];
        double side = v[vp], coeff = 0.0;
        for (int q = 0; q < len; ++q) {
          const int c2 = id[ip + 1 + q];
          const double a = v[vp + 1 + q];
          if (c2 == col) coeff = a; else side -= a * x[c2];
        }
        const double cand = side / coeff;
        ext = pos ? fmax(ext, cand) : fmin(ext, cand);
        ip += len + 1;
        vp += len + 1;
      }
      x[col] = ext;
    }
    if (dual && z) { z[col] = 0.0; s.got[col] = 1; }
  } else if (type == kFmeCol) {
    // replay_projected_column (postsolve_projected_variables.cuh:10-66):
    // x = max of the lower expressions (else min of the upper ones, else 0);
    // the column's reduced cost and its rows' duals are zero.
    const int K = id[0], col = id[1], L = id[3 + K];
    int64_t meta = 4 + K, at = 4 + K + 2 * int64_t(L), vp = 0;
    if (primal) {
      double lo = -INFINITY, hi = INFINITY;
      bool has_lo = false, has_hi = false;
      for (int e = 0; e < L; ++e) {
        const int orient = id[meta++];
        const int len = id[meta++];
        double cand = v[vp];
        for (int t = 0; t < len; ++t) cand += v[vp + 1 + t] * x[id[at++]];
        if (orient > 0) { lo = fmax(lo, cand); has_lo = true; } else { hi = fmin(hi, cand); has_hi = true; }
        vp += 1 + len;
      }
      x[col] = has_lo ? lo : (has_hi ? hi : 0.0);
    }
    if (dual && z) { z[col] = 0.0; s.got[col] = 1; }
    if (dual && y) for (int t = 0; t < K; ++t) y[id[2 + t]] = 0.0;
  } else if (dual && type == kRowDualShift) {
    if (y) y[id[0]] += v[0];
  } else if (dual && type == kParallelRow && ni >= 2 && nv >= 5) {
    // replay_parallel_row (postsolve_parallel_rows.cuh:170-250).
    const int kept = id[0], del = id[1];
    const double r = v[0], kal = v[1], kau = v[2], dal = v[3], dau = v[4];
    if (fabs(r) <= tol || !y) return;
    double dsl = dal * r, dsu = dau * r;
    if (r < 0.0) { const double t = dsl; dsl = dsu; dsu = t; }
    if (dsl <= kal + tol && kau <= dsu + tol) { y[del] = 0.0; return; }
    if (!M.present) return;
    auto act = [&](int row) {
      double a = 0.0;
      for (offset_t q = M.A_ptr[row]; q < M.A_ptr[row + 1]; ++q) a += M.A_val[q] * x[M.A_idx[q]];
      return a;
    };
    auto state = [&](double a, double lo, double hi) {
      const bool L = pfin(lo) && a <= lo + tol, U = pfin(hi) && a >= hi - tol;
      return L && U ? 3 : L ? 1 : U ? 2 : 0;
    };
    const int ks = state(act(kept), kal, kau), ds = state(act(del), dal, dau);
    double ydl, ydh, ypl, yph;
    if (ds == 3) { ydl = -INFINITY; ydh = INFINITY; } else if (ds == 1) { ydl = 0.0; ydh = INFINITY; }
    else if (ds == 2) { ydl = -INFINITY; ydh = 0.0; } else { ydl = 0.0; ydh = 0.0; }
    const double pv = r * y[kept];
    if (ks == 3) { ypl = -INFINITY; yph = INFINITY; }
    else if (ks == 0) { ypl = pv; yph = pv; }
    else if (ks == 1) { if (r > 0.0) { ypl = -INFINITY; yph = pv; } else { ypl = pv; yph = INFINITY; } }
    else { if (r > 0.0) { ypl = pv; yph = INFINITY; } else { ypl = -INFINITY; yph = pv; } }
    const double sl = fmax(ydl, ypl), sh = fmin(ydh, yph);
    if (sl <= sh + tol) {
      const double yd = clamp_inf(0.0, sl, sh);
      y[kept] = y[kept] - yd / r;
      y[del] = yd;
      return;
    }
    const double yb = y[kept];
    double yp = yb, yd = 0.0;
    bool ok;
    if (fabs(yb) <= tol) { yp = 0.0; yd = 0.0; ok = true; }
    else {
      const double bl = fmax(kal, dsl), bu = fmin(kau, dsu);
      if (!(bl <= bu + tol)) ok = false;
      else {
        const bool lt = bl > kal + tol, ut = bu < kau - tol;
        if (lt && ut) ok = false;
        else if (!lt && !ut) { yp = yb; yd = 0.0; ok = true; }
        else {
          ok = true;
          if (yb > 0.0) { if (lt) { yp = 0.0; yd = r * yb; } else { yp = yb; yd = 0.0; } }
          else { if (lt) { yp = yb; yd = 0.0; } else { yp = 0.0; yd = r * yb; } }
        }
      }
    }
    if (ok) { y[kept] = yp; y[del] = yd; }
  } else if (dual && type == kDeletedRow && M.present && ni >= 2 && nv >= 3) {
    // replay_deleted_singleton_row (postsolve_singleton_rows.cuh:8-96).
    const int row = id[0], col = id[1];
    const double oal = v[0], oau = v[1], a = v[2];
    if (fabs(a) <= tol) return;
    double g = M.c[col];
    for (offset_t q = M.AT_ptr[col]; q < M.AT_ptr[col + 1]; ++q)
      if (M.AT_idx[q] != row && y) g -= M.AT_val[q] * y[M.AT_idx[q]];
    const double xj = x[col], zb = z[col], ra = a * xj;
    const bool rl = isfinite(oal) && ra <= oal + tol, ru = isfinite(oau) && ra >= oau - tol;
    double lo = -INFINITY, hi = INFINITY;
    if (!(rl && ru)) {
      if (rl) { if (a > 0.0) hi = g; else lo = g; }
      else if (ru) { if (a > 0.0) lo = g; else hi = g; }
      else { lo = g; hi = g; }
    }
    const bool L = at_lower(xj, M.l[col], tol), U = at_upper(xj, M.u[col], tol);
    double zl = lo, zh = hi;
    if (!L && !U) {
      if ((isfinite(lo) && lo > tol) || (isfinite(hi) && hi < -tol)) { zl = g; zh = g; } else { zl = 0.0; zh = 0.0; }
    } else if (L && !U) zl = fmax(zl, 0.0);
    else if (!L && U) zh = fmin(zh, 0.0);
    if (isfinite(zl) && isfinite(zh) && zl > zh + tol) return;
    const double zn = clamp_inf(zb, zl, zh);
    z[col] = zn;
    if (y) y[row] = (g - zn) / a;
    s.got[col] = 1;
  } else if (dual && type == kRowImpliedBoundChange && M.present && ni >= 2) {
    // replay_row_implied_bound_change (postsolve_bound_strengthening.cuh:8-76).
    const int col = id[0], row = id[1];
    if (!s.got[col]) return;
    const double ol = v[0], ou = v[1], nl = v[2], nu = v[3];
    const bool lc = nl > ol + tol, uc = nu < ou - tol;
    if (lc == uc) return;
    const double ib = lc ? nl : nu, other = lc ? ou : ol;
    const bool other_lower = !lc;
    const double xj = x[col], zj = z[col];
    if (pfin(other) && fabs(xj - other) <= tol) {
      const bool ok = other_lower ? (zj >= -tol) : (zj <= tol);
      if (ok) return;
    }
    if (fabs(xj - ib) > tol) return;
    double aij = 0.0;
    for (offset_t q = M.A_ptr[row]; q < M.A_ptr[row + 1]; ++q)
      if (M.A_idx[q] == col) { aij = M.A_val[q]; break; }
    if (fabs(aij) <= tol) return;
    if (y) y[row] += zj / aij;
    for (offset_t q = M.A_ptr[row]; q < M.A_ptr[row + 1]; ++q) {
      const int kc = M.A_idx[q];
      if (kc == col || !s.got[kc]) continue;
      z[kc] -= (M.A_val[q] / aij) * zj;
    }
    z[col] = 0.0;
    s.got[col] = 1;
  }
}

struct SegView {
  const int32_t* types;
  const int64_t* is;
  const int64_t* vs;
  const int32_t* idx;
  const double* val;
  int64_t count;
};

// The reduced solution to original indices: x, z and the retrieval flag of a
// kept column, y of a kept row, in one launch.
__global__ void scatter_solution(Sol s, const double* __restrict__ x_red, const double* __restrict__ y_red,
                                 const double* __restrict__ z_red, const int32_t* __restrict__ rows, int32_t m,
                                 const int32_t* __restrict__ cols, int32_t n) {
  after_previous_kernel();
  const int top = n > m ? n : m;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < top; i += gridDim.x * blockDim.x) {
    if (i < n) {
      const int j = cols[i];
      if (x_red) s.x[j] = x_red[i];
      if (s.z && z_red) s.z[j] = z_red[i];
      s.got[j] = 1;
    }
    if (i < m && s.y && y_red) s.y[rows[i]] = y_red[i];
  }
}

// The fixed-value segments of a record, up to 64 a launch: a column is removed once, so
// it is in one of them at most and they can be restored together.
struct FixedViews {
  static constexpr int kMax = 64;
  int count;
  struct {
    const int32_t* idx;
    const double* val;
    int64_t count;
  } segment[kMax];
};
__global__ void restore_fixed(double* __restrict__ x, FixedViews fixed) {
  after_previous_kernel();
  for (int k = 0; k < fixed.count; ++k) {
    const auto& f = fixed.segment[k];
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < f.count; i += int64_t(gridDim.x) * blockDim.x)
      x[f.idx[i]] = f.val[i];
  }
}
// project_column_duals_from_original (gpu_postsolve.cu:355-398, postsolve_common.cuh:59-94):
// warp per column, A^T y summed sequentially by lane 0 in stored order.
__global__ void project_duals(int n, const uint8_t* __restrict__ prot, Model M, const double* __restrict__ x,
                              const double* __restrict__ y, double* __restrict__ z) {
  after_previous_kernel();
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    if (prot[j]) continue;
    double aty = 0.0;
    for (offset_t q = M.AT_ptr[j]; q < M.AT_ptr[j + 1]; ++q) aty += M.AT_val[q] * y[M.AT_idx[q]];
    const double r = M.c[j] - aty;
    const bool L = at_lower(x[j], M.l[j], kTol), U = at_upper(x[j], M.u[j], kTol);
    double zj;
    if (L && U) zj = r; else if (!L && !U) zj = 0.0; else if (L) zj = fmax(r, 0.0); else zj = fmin(r, 0.0);
    const double eps = fmin(kTol, 1.0e-12);
    if (zj > eps && !isfinite(M.l[j])) zj = 0.0;
    else if (zj < -eps && !isfinite(M.u[j])) zj = 0.0;
    z[j] = zj;
  }
}

SegView view(const PostsolveSegment& s) { return {s.types.p, s.is.p, s.vs.p, s.idx.p, s.val.p, s.count}; }

// ---- component-parallel replay ----------------------------------------------
//
// Replaying the tape in reverse chronological order is equivalent to
// replaying, in that order, each group of records that share a resource one
// of them writes, with the groups independent of one another.  Resources are
// the columns (x, z and the retrieval flag together) and the rows (y) of the
// original model; per pass only what that pass reads or writes counts (x is
// read-only in the dual pass, y and z untouched in the primal pass).  Records
// that do nothing in a pass (variable bound changes, the dual-only records in
// the primal pass, records whose own values and x show that they change
// nothing) drop out.  Groups come from a lock-free union-find over the
// records.

struct TapeView {
  const SegView* segs;       // device array
  const int64_t* starts;     // global index of each segment's first record
  int nseg;
  int64_t total;
  __device__ void at(int64_t g, int& type, const int32_t*& id, int64_t& ni, const double*& v, int64_t& nv) const {
    int lo = 0, hi = nseg - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (starts[mid] <= g) lo = mid; else hi = mid - 1;
    }
    const SegView& t = segs[lo];
    const int64_t k = g - starts[lo];
    type = t.types[k];
    id = t.idx + t.is[k];
    ni = t.is[k + 1] - t.is[k];
    v = t.val + t.vs[k];
    nv = t.vs[k + 1] - t.vs[k];
  }
};

__device__ __forceinline__ bool replays_in(int type, bool dual) {
  if (type == kFixedVariable || type == kInfiniteBoundDualFix || type == kSingletonColumnSubstitution ||
      type == kParallelColumn || type == kDoubletonEquation || type == kFmeCol)
    return true;
  return dual && (type == kRowDualShift || type == kParallelRow || type == kDeletedRow || type == kRowImpliedBoundChange);
}

// A record that replay_record leaves without a write whatever z, y and the
// retrieval flags hold.  A row-implied bound change acts only if exactly one
// of its bounds moved and x sits at the implied one (x is final before the
// dual pass).  At a point off the bounds almost none does, while each would tie
// all columns of its row into one group: on the QAP N = 30 relaxation the 0.8M
// records formed one group that a single thread replayed in 1,325 ms; without
// the records that cannot act the whole call (presolve and postsolve) takes
// 7.2 ms, 1,306 ms before.  At a point on the bounds, as a solver's is, they act
// and the groups stay: the QAP N = 12 relaxation's postsolve takes 0.1 ms for a
// point off all bounds (29.6 before), 36 ms with half of x on them (49) and 57
// ms with all (66).
__device__ __forceinline__ bool acts_in_dual(int type, const int32_t* id, int64_t ni, const double* v,
                                             const Model& M, const double* x) {
  if (type != kRowImpliedBoundChange) return true;
  if (!M.present || ni < 2) return false;
  const bool lc = v[2] > v[0] + kTol, uc = v[3] < v[1] - kTol;
  if (lc == uc) return false;
  return !(fabs(x[id[0]] - (lc ? v[2] : v[3])) > kTol);
}

// Calls visit(resource, writes) for every resource the record touches in the
// pass; columns are 0..n-1, rows n..n+m-1.
template <class F>
__device__ void record_resources(int type, const int32_t* id, int64_t ni, int64_t nv, bool dual, int m, int n,
                                 const Model& M, F visit) {
  auto col = [&](int j, bool w) { if (j >= 0 && j < n) visit(j, w); };
  auto row = [&](int i, bool w) { if (i >= 0 && i < m) visit(n + i, w); };
  if (!dual) {
    switch (type) {
      case kFixedVariable: col(id[0], true); break;
      case kInfiniteBoundDualFix: {
        col(id[1], true);
        int64_t ip = 3;
        for (int r = 0; r < id[2] && ip < ni; ++r) {
          const int len = id[ip];
          for (int q = 0; q < len && ip + 1 + q < ni; ++q) col(id[ip + 1 + q], false);
          ip += len + 1;
        }
        break;
      }
      case kSingletonColumnSubstitution:
        col(id[0], true);
        for (int q = 0; q < id[2] && 3 + q < ni; ++q) col(id[3 + q], false);
        break;
      case kParallelColumn: col(id[0], true); col(id[1], true); break;
      case kDoubletonEquation: col(id[0], true); col(id[1], false); break;
      case kFmeCol:
        if (ni >= 4) {
          const int K = id[0];
          col(id[1], true);
          if (3 + K < ni) {
            const int terms = id[2 + K];
            const int64_t first = int64_t(4 + K) + 2 * int64_t(id[3 + K]);
            for (int t = 0; t < terms && first + t < ni; ++t) col(id[first + t], false);
          }
        }
        break;
      default: break;
    }
    return;
  }
  switch (type) {
    case kFixedVariable:
      col(id[0], true);
      for (int64_t q = 1; q < ni; ++q) row(id[q], false);
      break;
    case kInfiniteBoundDualFix: col(id[1], true); break;
    case kSingletonColumnSubstitution: col(id[0], true); row(id[1], true); break;
    case kParallelColumn: col(id[0], true); col(id[1], false); break;
    case kDoubletonEquation:
      col(id[0], true); col(id[1], true); row(id[2], true);
      if (ni >= 4 && nv >= 12) {
        for (int q = 0; q < id[3] && 4 + q < ni; ++q) row(id[4 + q], false);
      } else if (M.present && id[0] >= 0 && id[0] < n) {
        for (offset_t q = M.AT_ptr[id[0]]; q < M.AT_ptr[id[0] + 1]; ++q) row(M.AT_idx[q], false);
      }
      break;
    case kFmeCol:
      if (ni >= 2) {
        col(id[1], true);
        for (int t = 0; t < id[0] && 2 + t < ni; ++t) row(id[2 + t], true);
      }
      break;
    case kRowDualShift: row(id[0], true); break;
    case kParallelRow: if (ni >= 2) { row(id[0], true); row(id[1], true); } break;
    case kDeletedRow:
      if (ni >= 2) {
        row(id[0], true); col(id[1], true);
        if (M.present && id[1] >= 0 && id[1] < n)
          for (offset_t q = M.AT_ptr[id[1]]; q < M.AT_ptr[id[1] + 1]; ++q) row(M.AT_idx[q], false);
      }
      break;
    case kRowImpliedBoundChange:
      if (ni >= 2) {
        col(id[0], true); row(id[1], true);
        if (M.present && id[1] >= 0 && id[1] < m)
          for (offset_t q = M.A_ptr[id[1]]; q < M.A_ptr[id[1] + 1]; ++q) col(M.A_idx[q], true);
      }
      break;
    default: break;
  }
}

// A record that a pass replays.
__device__ __forceinline__ bool record_acts(int type, const int32_t* id, int64_t ni, const double* v, bool dual,
                                            const Model& M, const double* x) {
  return replays_in(type, dual) && (!dual || acts_in_dual(type, id, ni, v, M, x));
}

// Root of a record's group; the path is halved on the way (a store to a
// record that is no root, which no link ever targets).
__device__ __forceinline__ int uf_root(int32_t* parent, int a) {
  volatile int32_t* p = parent;
  for (;;) {
    const int b = p[a];
    if (b == a) return a;
    const int c = p[b];
    if (c == b) return b;
    p[a] = c;
    a = c;
  }
}
// Link the larger root under the smaller; a failed CAS means the root moved,
// so retry from the new roots.  Links always point to smaller indices, so no
// cycle can form and every retry makes progress.
__device__ void uf_unite(int32_t* parent, int a, int b) {
  for (;;) {
    a = uf_root(parent, a);
    b = uf_root(parent, b);
    if (a == b) return;
    const int hi = a > b ? a : b, lo = a > b ? b : a;
    if (atomicCAS(parent + hi, hi, lo) == hi) return;
  }
}

// One record of the tape.
struct RecordAt {
  int type;
  const int32_t* id;
  int64_t ni, nv;
  const double* v;
  __device__ RecordAt(const TapeView& t, int64_t g) { t.at(g, type, id, ni, v, nv); }
};

// Records lo + q, q < count, of the tape.  First every record that acts
// claims the resources it writes (owner: record + 1, 0 for none); the others
// get parent -1.
__device__ __forceinline__ void claim_record(const TapeView& t, int64_t lo, int q, bool dual, int m, int n,
                                             const Model& M, const double* x, int32_t* owner, int32_t* parent) {
  const RecordAt r(t, lo + q);
  const bool acts = record_acts(r.type, r.id, r.ni, r.v, dual, M, x);
  parent[q] = acts ? q : -1;
  if (acts)
    record_resources(r.type, r.id, r.ni, r.nv, dual, m, n, M, [&](int res, bool w) {
      if (w && owner[res] == 0) atomicCAS(owner + res, 0, q + 1);
    });
}
// Then every record joins the owner of each resource it touches.
__device__ __forceinline__ void connect_record(const TapeView& t, int64_t lo, int q, bool dual, int m, int n,
                                               const Model& M, const int32_t* owner, int32_t* parent) {
  if (parent[q] < 0) return;
  const RecordAt r(t, lo + q);
  record_resources(r.type, r.id, r.ni, r.nv, dual, m, n, M, [&](int res, bool) {
    const int o = owner[res] - 1;
    if (o >= 0 && o != q) uf_unite(parent, q, o);
  });
}
__device__ __forceinline__ void replay_at(const TapeView& t, int64_t g, const Sol& s, const Model& M, bool dual) {
  const RecordAt r(t, g);
  replay_record(r.type, r.id, r.ni, r.v, r.nv, s, M, !dual, dual);
}

__global__ void rg_claim(TapeView t, int64_t lo, int count, int dual, int m, int n, Model M,
                         const double* __restrict__ x, int32_t* owner, int32_t* __restrict__ parent) {
  after_previous_kernel();
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x)
    claim_record(t, lo, q, dual != 0, m, n, M, x, owner, parent);
}
__global__ void rg_connect(TapeView t, int64_t lo, int count, int dual, int m, int n, Model M,
                           const int32_t* __restrict__ owner, int32_t* parent) {
  after_previous_kernel();
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x)
    connect_record(t, lo, q, dual != 0, m, n, M, owner, parent);
}
// Roots are final: a root with another member is marked.
__global__ void rg_roots(int count, int32_t* parent, uint8_t* __restrict__ shared_root) {
  after_previous_kernel();
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x) {
    if (parent[q] < 0) continue;
    const int r = uf_root(parent, q);
    if (r != q) shared_root[r] = 1;
  }
}
// A record alone in its group is replayed here; the members of larger groups
// are listed as (root, record) for the sort.  Most records are alone, so the
// sort sees few, and the whole tape needs one wait per pass (500,000 x
// 1,250,000 random LP: 862 us before, with every record sorted, four waits
// and one marking launch per segment; 272 us now).
__global__ void __launch_bounds__(kThreads) rg_replay_alone(TapeView t, int64_t lo, int count, int dual, Sol s, Model M,
                                                            int32_t* parent, const uint8_t* __restrict__ shared_root,
                                                            uint64_t* __restrict__ keys, int32_t* __restrict__ vals,
                                                            Report report) {
  after_previous_kernel();
  const int stride = gridDim.x * blockDim.x;
  const int64_t top = (int64_t(count) + stride - 1) / stride * stride;
  for (int64_t p = blockIdx.x * blockDim.x + threadIdx.x; p < top; p += stride) {
    const int q = int(p);
    const int r = p < count && parent[q] >= 0 ? uf_root(parent, q) : -1;
    const bool listed = r >= 0 && (r != q || shared_root[q]);
    const int at = block_append(report.words, listed);
    if (listed) {
      keys[at] = (uint64_t(uint32_t(r)) << 32) | uint32_t(q);
      vals[at] = q;
    } else if (r >= 0) {
      replay_at(t, lo + q, s, M, dual != 0);
    }
  }
  post_report(report);
}
// One thread per listed group: the thread at the group's last (newest) record
// replays it and walks back to the group's first.
__global__ void rg_replay_groups(TapeView t, int64_t lo, int listed, const uint64_t* __restrict__ keys, int dual, Sol s,
                                 Model M) {
  after_previous_kernel();
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < listed; e += gridDim.x * blockDim.x) {
    const uint32_t root = uint32_t(keys[e] >> 32);
    if (e + 1 < listed && uint32_t(keys[e + 1] >> 32) == root) continue;
    for (int q = e; q >= 0; --q) {
      const uint64_t k = keys[q];
      if (uint32_t(k >> 32) != root) break;
      replay_at(t, lo + int64_t(uint32_t(k)), s, M, dual != 0);
    }
  }
}

// Tapes of at most kBlockTape records: the whole replay, both passes, in one
// block, with the union-find and the sort in shared memory.  A tape this
// short is bound by launches: the passes above cost about eight launches and
// a wait each, and one thread alone walks a record in 1-2 us (the 400 x 1,000
// slack LP's tape took 0.47 ms; with the block its call went from 7.1 to
// 6.5 ms).  A record's entries are walked by one thread, three times a pass, so
// past one record a thread the grid's threads are worth more than the launches
// once the records are long: 1,000 records of 23, 43, 163 and 323 entries take 130,
// 168, 437 and 766 us in the block and about 130, 143, 236 and 358 us on the grid.
// The line is drawn on the entries walked: the tape's indices, and a row or column
// of the model for each record, which some types walk.
constexpr int kBlockTape = 2048;
constexpr double kBlockTapeEntries = 65536.0;
constexpr int kBlockReplayThreads = 512;
__global__ void __launch_bounds__(kBlockReplayThreads)
replay_block(TapeView t, int64_t lo, int count, int primal, int dual, int m, int n, Sol s, Model M, int32_t* owner) {
  after_previous_kernel();
  __shared__ int32_t parent[kBlockTape];
  __shared__ uint32_t key[kBlockTape];
  __shared__ uint8_t shared_root[kBlockTape];
  __shared__ int listed;
  for (int pass = primal ? 0 : 1; pass < (dual ? 2 : 1); ++pass) {
    const bool d = pass == 1;
    if (threadIdx.x == 0) listed = 0;
    for (int q = threadIdx.x; q < count; q += kBlockReplayThreads) {
      shared_root[q] = 0;
      claim_record(t, lo, q, d, m, n, M, s.x, owner, parent);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < count; q += kBlockReplayThreads) connect_record(t, lo, q, d, m, n, M, owner, parent);
    __syncthreads();
    for (int q = threadIdx.x; q < count; q += kBlockReplayThreads) {
      if (parent[q] < 0) continue;
      const int r = uf_root(parent, q);
      if (r != q) shared_root[r] = 1;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < count; q += kBlockReplayThreads) {
      if (parent[q] < 0) continue;
      if (!d && dual) {   // the dual pass claims afresh
        const RecordAt r(t, lo + q);
        record_resources(r.type, r.id, r.ni, r.nv, d, m, n, M, [&](int res, bool w) { if (w) owner[res] = 0; });
      }
      const int root = uf_root(parent, q);
      if (root != q || shared_root[q]) key[atomicAdd(&listed, 1)] = (uint32_t(root) << 16) | uint32_t(q);
      else replay_at(t, lo + q, s, M, d);
    }
    __syncthreads();
    int size = 1;
    while (size < listed) size <<= 1;
    for (int i = listed + int(threadIdx.x); i < size; i += kBlockReplayThreads) key[i] = 0xffffffffu;
    __syncthreads();
    for (int width = 2; width <= size; width <<= 1)
      for (int stride = width >> 1; stride > 0; stride >>= 1) {
        for (int i = threadIdx.x; i < size; i += kBlockReplayThreads) {
          const int j = i ^ stride;
          const uint32_t a = key[i], b = j > i ? key[j] : a;
          if (j > i && (a > b) == ((i & width) == 0)) {
            key[i] = b;
            key[j] = a;
          }
        }
        __syncthreads();
      }
    for (int e = threadIdx.x; e < listed; e += kBlockReplayThreads) {
      const uint32_t root = key[e] >> 16;
      if (e + 1 < listed && key[e + 1] >> 16 == root) continue;
      for (int q = e; q >= 0 && key[q] >> 16 == root; --q) replay_at(t, lo + int64_t(key[q] & 0xffffu), s, M, d);
    }
    __syncthreads();
  }
}

// Replays the records [lo, hi) of the whole tape (global indices): the primal
// pass, the dual pass or both.  A record walks about `entries` entries.
void replay_range(const TapeView& t, double entries, int m0, int n0, const Sol& s, const Model& M, bool primal,
                  bool dual, cudaStream_t st, int64_t lo, int64_t hi) {
  if (lo >= hi) return;
  if (hi - lo > INT32_MAX) throw LengthError("postsolve: more than 2^31 - 1 tape records");
  const int count = int(hi - lo);
  const size_t resources = size_t(m0) + size_t(n0);
  if (count <= kBlockReplayThreads || (count <= kBlockTape && entries * count <= kBlockTapeEntries)) {
    DBuf<int32_t> owner(std::max<size_t>(resources, 1), st);
    owner.zero();
    GPP_LAUNCH(replay_block, 1, kBlockReplayThreads, 0, st, t, lo, count, int(primal), int(dual), m0, n0, s, M,
               owner.p);
    return;
  }
  // Owners and the marks of shared roots, cleared at once.
  DBuf<int32_t> scratch(resources + (size_t(count) + 3) / 4, st);
  int32_t* owner = scratch.p;
  auto* shared_root = reinterpret_cast<uint8_t*>(owner + resources);
  DBuf<int32_t> parent(size_t(count), st), vals(size_t(count), st);
  DBuf<uint64_t> keys(size_t(count), st);
  const int g = grid_stride_blocks(count);
  for (int pass = primal ? 0 : 1; pass < (dual ? 2 : 1); ++pass) {
    scratch.zero();
    GPP_LAUNCH(rg_claim, g, kThreads, 0, st, t, lo, count, pass, m0, n0, M, s.x, owner, parent.p);
    GPP_LAUNCH(rg_connect, g, kThreads, 0, st, t, lo, count, pass, m0, n0, M, owner, parent.p);
    GPP_LAUNCH(rg_roots, g, kThreads, 0, st, count, parent.p, shared_root);
    const Report report = ctx().open_report(1);
    GPP_LAUNCH(rg_replay_alone, g, kThreads, 0, st, t, lo, count, pass, s, M, parent.p, shared_root, keys.p, vals.p,
               report);
    const int listed = int(ctx().await(report)[0]);
    if (!listed) continue;
    radix_sort_pairs(keys.p, vals.p, listed, st, (bits_up_to(count - 1) << 32) | bits_up_to(count - 1));
    GPP_LAUNCH(rg_replay_groups, grid_stride_blocks(listed), kThreads, 0, st, t, lo, listed, keys.p, pass, s, M);
  }
}

__global__ void mark_protected(TapeView t, uint8_t* __restrict__ prot, int n) {
  after_previous_kernel();
  for (int64_t g = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; g < t.total; g += int64_t(gridDim.x) * blockDim.x) {
    const RecordAt r(t, g);
    int a = -1, b = -1;
    if (r.type == kSingletonColumnSubstitution || r.type == kParallelColumn) a = r.id[0];
    if (r.type == kDoubletonEquation) { a = r.id[0]; b = r.id[1]; }
    if (r.type == kInfiniteBoundDualFix) a = r.id[1];
    if (a >= 0 && a < n) prot[a] = 1;
    if (b >= 0 && b < n) prot[b] = 1;
  }
}

// ---- piecewise-linear primal recoveries ---------------------------------------
// postsolve_piecewise_linear_reformulation_absolute_value.cu:9-105.

__global__ void restore_splits(double* __restrict__ x, const int32_t* __restrict__ t, const int32_t* __restrict__ e,
                               const double* __restrict__ rho, int k) {
  after_previous_kernel();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k; i += gridDim.x * blockDim.x) {
    const double tv = x[t[i]], ev = x[e[i]];
    x[t[i]] = tv + ev;
    x[e[i]] = (tv - ev) / rho[i];
  }
}
__global__ void restore_pairs(double* __restrict__ x, const int32_t* __restrict__ bound,
                              const int32_t* __restrict__ free_col, int k) {
  after_previous_kernel();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k; i += gridDim.x * blockDim.x) x[free_col[i]] = x[bound[i]];
}
__global__ void restore_links(double* __restrict__ x, const int32_t* __restrict__ slack, const int32_t* __restrict__ t,
                              const double* __restrict__ f, int k) {
  after_previous_kernel();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k; i += gridDim.x * blockDim.x) x[slack[i]] = f[i] * x[t[i]];
}
// One warp per group: slack = max(l_slack (0 when absent or not finite),
// max_k factor_k t_k).  fmax ignores NaN and is exact, so any order of the
// maximum gives the reference's value.
__global__ void restore_max_slacks(double* __restrict__ x, const int32_t* __restrict__ slack,
                                   const int32_t* __restrict__ start, const int32_t* __restrict__ t,
                                   const double* __restrict__ f, int groups, const double* __restrict__ lower) {
  after_previous_kernel();
  const int lane = threadIdx.x & 31;
  for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < groups; g += (gridDim.x * blockDim.x) >> 5) {
    const int32_t sc = slack[g];
    double lb = lower ? lower[sc] : 0.0;
    if (!isfinite(lb)) lb = 0.0;
    double v = lb;
    for (int q = start[g] + lane; q < start[g + 1]; q += 32) v = fmax(v, f[q] * x[t[q]]);
    for (int o = 16; o; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) x[sc] = v;
  }
}

// Roots' values first, then every member (restore_piecewise_linear_reformulation_variable_pair,
// postsolve_piecewise_linear_reformulation_variable_pair.cu:9-95).
__global__ void cache_pair_roots(double* __restrict__ pc, double* __restrict__ mc, const double* __restrict__ x,
                                 const int32_t* __restrict__ rp, const int32_t* __restrict__ rm, int k) {
  after_previous_kernel();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k; i += gridDim.x * blockDim.x) {
    pc[i] = x[rp[i]];
    mc[i] = x[rm[i]];
  }
}
__global__ void restore_pair_members(double* __restrict__ x, const int32_t* __restrict__ plus,
                                     const int32_t* __restrict__ minus, const double* __restrict__ ps,
                                     const double* __restrict__ ms, const double* __restrict__ pc,
                                     const double* __restrict__ mc, int k) {
  after_previous_kernel();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k; i += gridDim.x * blockDim.x) {
    x[plus[i]] = ps[i] + pc[i];
    x[minus[i]] = ms[i] + mc[i];
  }
}

}  // namespace

void restore_variable_pair(double* x, const VarPairRecovery& r, cudaStream_t st) {
  if (!r.count) return;
  DBuf<double> pc(size_t(r.count), st), mc(size_t(r.count), st);
  GPP_LAUNCH(cache_pair_roots, grid_stride_blocks(r.count), kThreads, 0, st, pc.p, mc.p, x, r.root_plus.p,
             r.root_minus.p, r.count);
  GPP_LAUNCH(restore_pair_members, grid_stride_blocks(r.count), kThreads, 0, st, x, r.plus.p, r.minus.p,
             r.plus_shift.p, r.minus_shift.p, pc.p, mc.p, r.count);
}

void restore_absolute_value(double* x, const AbsValueRecovery& r, const double* lower, cudaStream_t st) {
  GPP_LAUNCH(restore_splits, grid_stride_blocks(r.splits), kThreads, 0, st, x, r.split_t.p, r.split_e.p,
             r.split_rho.p, r.splits);
  GPP_LAUNCH(restore_pairs, grid_stride_blocks(r.pairs), kThreads, 0, st, x, r.pair_bound.p, r.pair_free.p, r.pairs);
  GPP_LAUNCH(restore_links, grid_stride_blocks(r.links), kThreads, 0, st, x, r.link_slack.p, r.link_t.p,
             r.link_factor.p, r.links);
  GPP_LAUNCH(restore_max_slacks, grid_stride_blocks(int64_t(r.max_groups) * 32), kThreads, 0, st, x, r.max_slack.p,
             r.max_start.p, r.max_t.p, r.max_factor.p, r.max_groups, lower);
}

void run_postsolve(const PresolveOutput& out, const double* x_red, const double* y_red, const double* z_red,
                   const gpp_lp* original, double* x, double* y, double* z, const double* lower) {
  const NvtxRange range("postsolve");
  if (!lower && original) lower = original->l;
  auto st = ctx().stream;
  const Record& r = out.record;
  const int m0 = r.m0, n0 = r.n0;
  if (n0) check(cudaMemsetAsync(x, 0, sizeof(double) * n0, st), "clear x");
  if (m0 && y) check(cudaMemsetAsync(y, 0, sizeof(double) * m0, st), "clear y");
  if (n0 && z) check(cudaMemsetAsync(z, 0, sizeof(double) * n0, st), "clear z");
  // The retrieval flags, then the marks of columns whose z a record set.
  const size_t columns = size_t(std::max(n0, 1));
  DBuf<uint8_t> got(2 * columns, st);
  got.zero();
  uint8_t* prot = got.p + columns;
  const Sol s{x, y, z, got.p};
  if (r.n || r.m)
    GPP_LAUNCH(scatter_solution, grid_stride_blocks(std::max(r.n, r.m)), kThreads, 0, st, s, x_red, y_red, z_red,
               r.rows.p, r.m, r.cols.p, r.n);
  for (size_t first = 0; first < r.fixed.size();) {
    FixedViews v{};
    int64_t most = 0;
    for (; first < r.fixed.size() && v.count < FixedViews::kMax; ++first) {
      const FixedSegment& f = r.fixed[first];
      if (!f.count) continue;
      v.segment[v.count++] = {f.idx.p, f.val.p, f.count};
      most = std::max(most, f.count);
    }
    if (v.count) GPP_LAUNCH(restore_fixed, grid_stride_blocks(most), kThreads, 0, st, x, v);
  }
  // Views of the tape's segments and the global index of each one's first record,
  // uploaded together.
  std::vector<SegView> segs;
  std::vector<int64_t> starts;
  int64_t total = 0;
  for (const auto& seg : r.segments) {
    if (!seg.count) continue;
    segs.push_back(view(seg));
    starts.push_back(total);
    total += seg.count;
  }
  const size_t seg_bytes = sizeof(SegView) * segs.size(), start_bytes = sizeof(int64_t) * starts.size();
  std::vector<unsigned char> packed(seg_bytes + start_bytes);
  DBuf<unsigned char> views(packed.size(), st);
  if (!packed.empty()) {
    std::memcpy(packed.data(), segs.data(), seg_bytes);
    std::memcpy(packed.data() + seg_bytes, starts.data(), start_bytes);
    check(cudaMemcpyAsync(views.p, packed.data(), packed.size(), cudaMemcpyHostToDevice, st), "record views");
  }
  const TapeView t{reinterpret_cast<const SegView*>(views.p), reinterpret_cast<const int64_t*>(views.p + seg_bytes),
                   int(segs.size()), total};
  Model M{};
  if (original) {
    M = Model{original->A.rowPtr, original->AT.rowPtr, original->A.colVal, original->AT.colVal, original->A.nzVal,
              original->AT.nzVal, original->c, original->l, original->u, true};
  }
  // Primal pass split at the piecewise-linear checkpoints, newest first: the
  // records after a checkpoint, then its recovery (postsolve_gpu,
  // gpu_postsolve.cu:637-663); the dual pass over the whole tape.
  int64_t range_end = r.records;
  double entries = total ? double(r.indices) / double(total) : 0.0;
  if (original) entries += double(original->A.nnz) / std::max(1, std::min(m0, n0));
  for (auto it = r.timeline.rbegin(); it != r.timeline.rend(); ++it) {
    replay_range(t, entries, m0, n0, s, M, true, false, st, it->tape_position, range_end);
    if (it->kind == 0) restore_absolute_value(x, r.absval[size_t(it->payload)], lower, st);
    else restore_variable_pair(x, r.varpair[size_t(it->payload)], st);
    range_end = it->tape_position;
  }
  if (r.timeline.empty()) {
    replay_range(t, entries, m0, n0, s, M, true, true, st, 0, r.records);
  } else {
    replay_range(t, entries, m0, n0, s, M, true, false, st, 0, range_end);
    replay_range(t, entries, m0, n0, s, M, false, true, st, 0, r.records);
  }
  if (original && y && z && n0) {
    if (total) GPP_LAUNCH(mark_protected, grid_stride_blocks(total), kThreads, 0, st, t, prot, n0);
    GPP_LAUNCH(project_duals, grid_stride_blocks(n0), kThreads, 0, st, n0, prot, M, x, y, z);
  }
  ctx().sync("postsolve");
}

}  // namespace gpp

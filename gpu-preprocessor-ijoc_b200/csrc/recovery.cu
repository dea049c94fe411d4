// GPU-resident recovery record: original-index maps, fixed-value segments and
// the chronological postsolve tape.
//
// Reference: cpp/src/presolve/device_recovery.cu:42-276,881-1027.  Rules
// write records with the indices of the current (physical) model; capture
// rewrites them to original indices with the current maps, so the tape that
// postsolve replays is expressed in the original model throughout.
#include "engine.cuh"
#include "scan.cuh"

namespace gpp {

namespace {

__global__ void iota(int32_t* a, int32_t n) {
  after_previous_kernel();
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    a[i] = int32_t(i);
}

__device__ __forceinline__ int map_idx(int x, const int32_t* map, int n) { return x >= 0 && x < n ? map[x] : x; }

// Record types (the reference's PostsolveReductionType numbering).
enum : int {
  kFixedVariable = 0, kInfiniteBoundDualFix = 1, kSingletonColumnSubstitution = 2, kParallelColumn = 3,
  kParallelRow = 4, kDeletedRow = 5, kRowLowerBoundChange = 8, kRowUpperBoundChange = 9, kRowDualShift = 10,
  kVariableBoundChange = 11, kRowImpliedBoundChange = 12, kDoubletonEquation = 13, kFmeCol = 14
};

// The segments captured since the maps last changed, up to 32 a launch (a
// model's rounds leave two or three small ones each between two
// materialisations, 43 launches in a 50,000-column presolve).
struct SegmentViews {
  static constexpr int kMax = 32;
  int count;
  int64_t first[kMax + 1];   // records before the segment
  const int32_t* types[kMax];
  const int64_t* is[kMax];
  int32_t* idx[kMax];
};

// One thread per record; long supports are walked by the same thread (the
// records with long index lists are rare and bounded by the row length).
__global__ void globalize_kernel(SegmentViews v, const int32_t* __restrict__ rows, int m,
                                 const int32_t* __restrict__ cols, int n) {
  after_previous_kernel();
  const int64_t count = v.first[v.count];
  for (int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; r < count; r += int64_t(gridDim.x) * blockDim.x) {
    int s = 0;
    while (r >= v.first[s + 1]) ++s;
    const int64_t k = r - v.first[s];
    const int32_t* const types = v.types[s];
    const int64_t* const is = v.is[s];
    int32_t* id = v.idx[s] + is[k];
    const int64_t sz = is[k + 1] - is[k];
    switch (types[k]) {
      case kFixedVariable:
        if (sz) { id[0] = map_idx(id[0], cols, n); for (int64_t q = 1; q < sz; ++q) id[q] = map_idx(id[q], rows, m); }
        break;
      case kInfiniteBoundDualFix:
        if (sz >= 3) {
          id[1] = map_idx(id[1], cols, n);
          int64_t q = 3;
          while (q < sz) {
            const int len = id[q++];
            for (int r = 0; r < len && q < sz; ++r, ++q) id[q] = map_idx(id[q], cols, n);
          }
        }
        break;
      case kSingletonColumnSubstitution:
        if (sz >= 3) {
          id[0] = map_idx(id[0], cols, n);
          id[1] = map_idx(id[1], rows, m);
          for (int r = 0; r < id[2] && 3 + r < sz; ++r) id[3 + r] = map_idx(id[3 + r], cols, n);
        }
        break;
      case kParallelColumn:
        if (sz >= 2) { id[0] = map_idx(id[0], cols, n); id[1] = map_idx(id[1], cols, n); }
        break;
      case kParallelRow:
        if (sz >= 2) { id[0] = map_idx(id[0], rows, m); id[1] = map_idx(id[1], rows, m); }
        break;
      case kDeletedRow:
        if (sz) { id[0] = map_idx(id[0], rows, m); if (sz >= 2) id[1] = map_idx(id[1], cols, n); }
        break;
      case kRowLowerBoundChange: case kRowUpperBoundChange: case kRowDualShift:
        if (sz) id[0] = map_idx(id[0], rows, m);
        break;
      case kVariableBoundChange:
        if (sz) id[0] = map_idx(id[0], cols, n);
        break;
      case kRowImpliedBoundChange:
        if (sz >= 2) { id[0] = map_idx(id[0], cols, n); id[1] = map_idx(id[1], rows, m); }
        break;
      case kDoubletonEquation:
        if (sz >= 4) {
          id[0] = map_idx(id[0], cols, n);
          id[1] = map_idx(id[1], cols, n);
          id[2] = map_idx(id[2], rows, m);
          for (int r = 0; r < id[3] && 4 + r < sz; ++r) id[4 + r] = map_idx(id[4 + r], rows, m);
        }
        break;
      case kFmeCol:
        // [K, col, rows[K], terms, L, (orient, len)[L], cols[terms]].
        if (sz >= 4) {
          const int k_rows = id[0];
          id[1] = map_idx(id[1], cols, n);
          for (int r = 0; r < k_rows && 2 + r < sz; ++r) id[2 + r] = map_idx(id[2 + r], rows, m);
          if (3 + k_rows < sz) {
            const int terms = id[2 + k_rows], exprs = id[3 + k_rows];
            const int64_t first = int64_t(4 + k_rows) + 2 * int64_t(exprs);
            for (int t = 0; t < terms && first + t < sz; ++t) id[first + t] = map_idx(id[first + t], cols, n);
          }
        }
        break;
      default:
        break;
    }
  }
}

__global__ void globalize_ids(int32_t* __restrict__ ids, int64_t n, const int32_t* __restrict__ cols) {
  after_previous_kernel();
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    ids[i] = cols[ids[i]];
}

}  // namespace

void capture_absolute_value(Record& r, AbsValueRecovery&& step) {
  // update_device_recovery (device_recovery.cu:912-928): column ids through
  // the record's current map, a checkpoint at the current tape length.
  auto s = ctx().stream;
  auto glob = [&](DBuf<int32_t>& ids, int64_t n) {
    GPP_LAUNCH(globalize_ids, grid_stride_blocks(n), kThreads, 0, s, ids.p, n, r.cols.p);
  };
  glob(step.split_t, step.splits);
  glob(step.split_e, step.splits);
  glob(step.pair_bound, step.pairs);
  glob(step.pair_free, step.pairs);
  glob(step.link_slack, step.links);
  glob(step.link_t, step.links);
  glob(step.max_slack, step.max_groups);
  glob(step.max_t, step.max_entries);
  r.timeline.push_back(RecoveryCheckpoint{0, int32_t(r.absval.size()), r.records});
  r.absval.push_back(std::move(step));
}

void capture_variable_pair(Record& r, VarPairRecovery&& step) {
  // update_device_recovery (device_recovery.cu:929-941).
  auto s = ctx().stream;
  for (DBuf<int32_t>* ids : {&step.plus, &step.minus, &step.root_plus, &step.root_minus})
    GPP_LAUNCH(globalize_ids, grid_stride_blocks(step.count), kThreads, 0, s, ids->p, step.count, r.cols.p);
  r.timeline.push_back(RecoveryCheckpoint{1, int32_t(r.varpair.size()), r.records});
  r.varpair.push_back(std::move(step));
}

void init_record(Record& r, int32_t m, int32_t n) {
  auto s = ctx().stream;
  r.m0 = r.m = m;
  r.n0 = r.n = n;
  r.rows.alloc(size_t(m), s);
  r.cols.alloc(size_t(n), s);
  GPP_LAUNCH(iota, grid_stride_blocks(m), kThreads, 0, s, r.rows.p, m);
  GPP_LAUNCH(iota, grid_stride_blocks(n), kThreads, 0, s, r.cols.p, n);
}

PostsolveSegment make_segment(int64_t count, int64_t n_idx, int64_t n_val) {
  auto s = ctx().stream;
  PostsolveSegment seg;
  seg.count = count;
  seg.n_idx = n_idx;
  seg.n_val = n_val;
  seg.types.alloc(size_t(count), s);
  seg.is.alloc(size_t(count) + 1, s);
  seg.vs.alloc(size_t(count) + 1, s);
  seg.idx.alloc(size_t(n_idx), s);
  seg.val.alloc(size_t(n_val), s);
  return seg;
}

void globalize_segments(Record& r) {
  while (r.globalized < r.segments.size()) {
    SegmentViews v{};
    for (; v.count < SegmentViews::kMax && r.globalized < r.segments.size(); ++v.count, ++r.globalized) {
      PostsolveSegment& seg = r.segments[r.globalized];
      v.types[v.count] = seg.types.p;
      v.is[v.count] = seg.is.p;
      v.idx[v.count] = seg.idx.p;
      v.first[v.count + 1] = v.first[v.count] + seg.count;
    }
    GPP_LAUNCH(globalize_kernel, grid_stride_blocks(v.first[v.count]), kThreads, 0, ctx().stream, v, r.rows.p, r.m,
               r.cols.p, r.n);
  }
}

void capture_tape(Record& r, std::vector<PostsolveSegment>& tape) {
  for (auto& seg : tape) {
    if (!seg.count) continue;
    r.records += seg.count;
    r.indices += seg.n_idx;
    r.values += seg.n_val;
    r.segments.push_back(std::move(seg));
  }
  tape.clear();
}

void settle_fixed(Record& r) {
  auto& late = r.late_fixed;
  if (!late.open) return;
  auto& c = ctx();
  late.open = false;
  const int64_t count = c.await(c.fixed_mail, late.seq, "append_fixed")[0];
  if (count) {
    FixedSegment f;
    f.count = count;
    f.idx.alloc(size_t(count), c.stream);
    f.val.alloc(size_t(count), c.stream);
    f.idx.copy_from(late.idx.p, size_t(count));
    f.val.copy_from(late.val.p, size_t(count));
    r.fixed.push_back(std::move(f));
  }
  late.idx.release();
  late.val.release();
}

void append_fixed(Record& r, const uint8_t* keep_col, const uint8_t* prior, const double* l, const double* u,
                  int32_t n) {
  // append_fixed (device_recovery.cu:233-276).
  if (!n) return;
  settle_fixed(r);
  auto s = ctx().stream;
  // One selection over the columns finds the fixed ones and packs them (into
  // arrays for all columns, as their number is not known yet); the segment
  // keeps the packed part, once the next call or the presolve's end has read the
  // number without a wait of its own.
  auto& late = r.late_fixed;
  late.idx.alloc(size_t(n), s);
  late.val.alloc(size_t(n), s);
  late.seq = ctx().open_mail();
  late.open = true;
  const int32_t* cols = r.cols.p;
  int32_t* out_idx = late.idx.p;
  double* out_val = late.val.p;
  select_and_post(
      n,
      [=] __device__(int64_t i) {
        return (!prior || prior[i]) && !keep_col[i] && isfinite(l[i]) && isfinite(u[i]) && fabs(l[i] - u[i]) <= 1e-9;
      },
      [=] __device__(int64_t i, int at, bool taken) {
        if (!taken) return;
        out_idx[at] = cols[i];
        out_val[at] = 0.5 * (l[i] + u[i]);
      },
      ctx().fixed_mail, late.seq, s);
}

}  // namespace gpp

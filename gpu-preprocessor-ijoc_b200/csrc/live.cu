// Live-structure kernels: row schedules, live statistics, row activity
// summaries and column max |a|.
//
// Reference: cpp/src/presolve/gpu_presolve_kernels.cu:96-517,744-809.
// Each kernel is ONE launch whose blocks split into three roles: a
// thread-per-row pass over short rows, warp-per-row over the medium queue and
// block-per-row over the long queue.  Masked traversals hand every lane the
// live entries with live rank == lane (mod width), exactly the sequence a
// physically compacted row would give, so the floating-point association of
// the activity sums is the reference's:
//   short  : sequential left-to-right sum,
//   medium : 32 lane partials, shfl_down tree 16,8,4,2,1 (own + peer),
//   long   : 256 lane partials, per-warp shfl tree 1,2,4,8,16 then warp
//            aggregates added in warp order (cub::BlockReduce default).
#include "engine.cuh"
#include "live_visit.cuh"

#include <array>
#include <atomic>

namespace gpp {

namespace {

__device__ __forceinline__ int row_len(const offset_t* ptr, const int32_t* live_deg, int row) {
  return live_deg ? live_deg[row] : int(ptr[row + 1] - ptr[row]);
}

__global__ void classify_rows(const offset_t* __restrict__ ptr, int m, const int32_t* __restrict__ live_deg,
                              int32_t* __restrict__ medium, int32_t* __restrict__ longq,
                              int32_t* __restrict__ counts) {
  after_previous_kernel();
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  const int len = row < m ? row_len(ptr, live_deg, row) : 0;
  for (int g = 0; g < 2; ++g) {
    const bool sel = row < m && (g == 0 ? (len > kShortRow && len <= kLongRow) : len > kLongRow);
    const int at = block_append(counts + g, sel);
    if (sel) (g == 0 ? medium : longq)[at] = row;
  }
}

template <class T>
__device__ __forceinline__ T warp_sum_down(T v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, off);
  return v;
}

// cub::BlockReduce<T,256>::Sum order; result valid in thread 0.
template <class T>
__device__ __forceinline__ T block_sum_cub_order(T v, T* warp_aggs) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const T peer = __shfl_down_sync(0xffffffffu, v, off);
    if (lane + off <= 31) v = v + peer;
  }
  if (lane == 0) warp_aggs[threadIdx.x >> 5] = v;
  __syncthreads();
  T total = v;
  if (threadIdx.x == 0) {
    total = warp_aggs[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) total = total + warp_aggs[w];
  }
  __syncthreads();
  return total;
}

template <bool Plain>
struct ActivityTerm {
  const int32_t* idx;
  const double* val;
  const double2* lu;
  double zero_tol;
  L2Hints hint;
  // The term of live stored entry p whose column bounds are b.
  __device__ __forceinline__ void operator()(offset_t p, double2 b, double& lo, double& hi, int& ni, int& pi) const {
    add(ld_stream(val + p, hint.stream), b, lo, hi, ni, pi);   // streamed once: keep L2 for the gathered bounds
  }
  __device__ __forceinline__ void add(double a, double2 b, double& lo, double& hi, int& ni, int& pi) const {
    if constexpr (Plain) {
      // Plain sums of the redundant-row test: infinities propagate.
      lo += a >= 0.0 ? a * b.x : a * b.y;
      hi += a >= 0.0 ? a * b.y : a * b.x;
      return;
    }
    if (fabs(a) <= zero_tol) return;
    const double tlo = a >= 0.0 ? a * b.x : a * b.y;
    const double thi = a >= 0.0 ? a * b.y : a * b.x;
    if (isfinite(tlo)) lo += tlo; else if (tlo < 0.0) ++ni;
    if (isfinite(thi)) hi += thi; else if (thi > 0.0) ++pi;
  }
  __device__ __forceinline__ double2 bounds(offset_t p) const {
    return ld_keep(lu + ld_stream(idx + p, hint.stream), hint.keep);
  }
  // One live entry as the reference's lane partial holds it when the lane
  // sees no other entry: 0.0 + term (or 0.0 when the term is skipped), plus
  // the infinite-term counts.
  __device__ __forceinline__ void slot(double a, double2 b, double& plo, double& phi, int& ni, int& pi) const {
    plo = 0.0;
    phi = 0.0;
    if constexpr (Plain) {
      plo = plo + (a >= 0.0 ? a * b.x : a * b.y);
      phi = phi + (a >= 0.0 ? a * b.y : a * b.x);
      return;
    }
    if (fabs(a) <= zero_tol) return;
    const double tlo = a >= 0.0 ? a * b.x : a * b.y;
    const double thi = a >= 0.0 ? a * b.y : a * b.x;
    if (isfinite(tlo)) plo = plo + tlo; else if (tlo < 0.0) ++ni;
    if (isfinite(thi)) phi = phi + thi; else if (thi > 0.0) ++pi;
  }
};

// Medium rows of at most 32 stored entries (most rows of the random family
// hold 9-32) take eight lanes each, four rows per warp.  For such a row the
// reference's warp association is fixed by live rank k alone: lane k holds
// p[k] = 0.0 + term k (0.0 past the live length), and the shfl_down tree
// 16,8,4,2,1 leaves in lane l < 8, after its first two steps,
// (p[l] + p[l+16]) + (p[l+8] + p[l+24]); the tree 4,2,1 over those eight
// lanes finishes the sum with the same roundings.  So lane l of a group forms
// exactly that value and the group runs the last three steps.  Terms are
// staged in shared memory at their live rank, so masked rows give the same
// sums.
constexpr int kGroupRowMax = 32;

// The test of one row from its plain sums (rule_infeasible_and_redundant_rows.cu:158-240).
// Its sides are loaded with the row's entries, ahead of the sums.
struct RowSides {
  double al, au;
  bool kept, tested;
  __device__ __forceinline__ RowSides(const RedundantTest& t, int row, const uint8_t* keep_row,
                                      const int32_t* live_deg)
      : al(t.AL[row]), au(t.AU[row]), kept(keep_row[row]), tested(kept && live_deg[row] > 1) {}
  __device__ __forceinline__ RowSides() : al(0.0), au(0.0), kept(false), tested(false) {}
};
__device__ __forceinline__ uint32_t redundant_test(const RedundantTest& t, int row, const RowSides& sides, double lo,
                                                   double hi) {
  uint32_t found = 0;
  uint8_t a = 0;
  const double al = sides.al, au = sides.au;
  if (sides.tested) {
    const bool lf = isfinite(al), uf = isfinite(au);
    if (!(lf && uf && fabs(au - al) <= t.tol)) {
      if ((lf && hi < al - t.tol) || (uf && lo > au + t.tol)) {
        found = 1u;
      } else {
        const bool li = !lf || lo >= al - t.tol, ui = !uf || hi <= au + t.tol;
        if (li && ui) { a = 1; found = 2u; }
        else if (lf && li) { a = 2; found = 4u; }
        else if (uf && ui) { a = 3; found = 4u; }
      }
    }
  }
  t.action[row] = a;
  t.kinds[row] = row_kind(sides.kept, al, au);
  return found;
}

// With Plain the kernel forms the redundant-row rule's sums, in which
// infinities propagate, and tests each row as soon as its sums stand; the sums
// themselves are not stored.
//
// Latency-bound (every warp waits for its gathers, the L2 at a third of its
// rate), so the registers are held to four blocks an SM.
enum class Sums { kFinite, kRecords, kPlain };
template <Sums Form>
__global__ void __launch_bounds__(kThreads, 4)
activity_kernel(int m, const offset_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                const double* __restrict__ val, const double2* __restrict__ lu, double zero_tol,
                const uint8_t* __restrict__ keep_row, const int32_t* __restrict__ live_deg,
                const int32_t* __restrict__ medium, const int32_t* __restrict__ longq,
                const int32_t* __restrict__ counts, int short_blocks, int medium_blocks,
                double* __restrict__ min_fin, double* __restrict__ max_fin, int32_t* __restrict__ min_inf,
                int32_t* __restrict__ max_inf, RowRecords records, RedundantTest test) {
  after_previous_kernel();
  constexpr bool Plain = Form == Sums::kPlain;
  __shared__ int slots[256];
  __shared__ int warp_counts[8];
  __shared__ double dagg[8];
  __shared__ int iagg[8];
  __shared__ double group_lo[(kThreads / 32) * 4 * kGroupRowMax];
  __shared__ double group_hi[(kThreads / 32) * 4 * kGroupRowMax];
  const ActivityTerm<Plain> term{idx, val, lu, zero_tol, l2_hints()};
  const auto live_at = [&](offset_t p) { return !removed_column(term.bounds(p)); };
  uint32_t found = 0;
  const auto sides_of = [&](int row) {
    if constexpr (Form != Sums::kFinite) return RowSides(test, row, keep_row, live_deg);
    else return 0;
  };
  const auto finish = [&](int row, const auto& sides, double lo, double hi, int ni, int pi) {
    if constexpr (Plain) {
      found |= redundant_test(test, row, sides, lo, hi);
    } else if constexpr (Form == Sums::kRecords) {
      records.flags[row] = uint8_t(min(ni, 3) | min(pi, 3) << 2 | (sides.tested ? kRowLive : 0));
      if (sides.tested) {
        records.sums[2 * int64_t(row)] = make_double2(sides.al, sides.au);
        records.sums[2 * int64_t(row) + 1] = make_double2(lo, hi);
      }
    } else {
      min_fin[row] = lo; max_fin[row] = hi;
      if (min_inf) { min_inf[row] = ni; max_inf[row] = pi; }
    }
  };
  const int b = blockIdx.x;
  if (b < short_blocks) {
    // The next row's pointers and live length are loaded one iteration ahead.
    const int stride = short_blocks * blockDim.x;
    int i_next = b * blockDim.x + threadIdx.x;
    offset_t first_next = i_next < m ? ptr[i_next] : 0, last_next = i_next < m ? ptr[i_next + 1] : 0;
    int len_next = i_next < m && live_deg ? live_deg[i_next] : int(last_next - first_next);
    for (int i = i_next; i < m; i += stride) {
      const offset_t first = first_next, last = last_next;
      const int len = len_next;
      i_next = i + stride;
      first_next = i_next < m ? ptr[i_next] : 0;
      last_next = i_next < m ? ptr[i_next + 1] : 0;
      len_next = i_next < m && live_deg ? live_deg[i_next] : int(last_next - first_next);
      if (len > kShortRow) continue;
      const auto sides = sides_of(i);
      double lo = 0.0, hi = 0.0;
      int ni = 0, pi = 0;
      if (keep_row && !keep_row[i]) {
      } else if (last - first <= kShortRow) {
        // All loads of the (at most 8) entries first, then the sequential sum.
        int col[kShortRow];
        double a[kShortRow];
        double2 bnd[kShortRow];
#pragma unroll
        for (int k = 0; k < kShortRow; ++k) {
          col[k] = first + k < last ? ld_stream(idx + first + k, term.hint.stream) : -1;
          a[k] = first + k < last ? ld_stream(val + first + k, term.hint.stream) : 0.0;
        }
#pragma unroll
        for (int k = 0; k < kShortRow; ++k)
          bnd[k] = col[k] >= 0 ? ld_keep(lu + col[k], term.hint.keep) : make_double2(0.0, 0.0);
#pragma unroll
        for (int k = 0; k < kShortRow; ++k)
          if (col[k] >= 0 && !removed_column(bnd[k])) term.add(a[k], bnd[k], lo, hi, ni, pi);
      } else {
        for (offset_t p = first; p < last; ++p) {
          const double2 bnd = term.bounds(p);
          if (!removed_column(bnd)) term(p, bnd, lo, hi, ni, pi);
        }
      }
      finish(i, sides, lo, hi, ni, pi);
    }
  } else if (b < short_blocks + medium_blocks) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = lane >> 3, gl = lane & 7;
    const int nwarps = medium_blocks * (kThreads / 32);
    const int count = counts[0];
    double* glo = group_lo + (warp * 4 + grp) * kGroupRowMax;
    double* ghi = group_hi + (warp * 4 + grp) * kGroupRowMax;
    const auto full_row = [&](int row) {
      const auto sides = sides_of(row);
      double lo = 0.0, hi = 0.0;
      int ni = 0, pi = 0;
      const offset_t first = ptr[row], last = ptr[row + 1];
      const bool all_live = live_deg && live_deg[row] == int(last - first);
      if (!keep_row || keep_row[row])
        live_visit_by<32>(first, last, all_live, live_at, slots + warp * 32, nullptr,
                          [&](offset_t p) { term(p, term.bounds(p), lo, hi, ni, pi); });
      lo = warp_sum_down(lo); hi = warp_sum_down(hi); ni = warp_sum_down(ni); pi = warp_sum_down(pi);
      if (lane == 0) finish(row, sides, lo, hi, ni, pi);
    };
    // The row ids and row pointers of later iterations are loaded ahead (the
    // queue entry two iterations ahead, the pointers one ahead), so each
    // iteration's critical path starts at its entries instead of at the queue.
    const int step = nwarps * 4;
    const int q_first = ((b - short_blocks) * (kThreads / 32) + warp) * 4 + grp;
    int row_next = q_first < count ? medium[q_first] : 0;
    int row_after = q_first + step < count ? medium[q_first + step] : 0;
    offset_t first_next = q_first < count ? ptr[row_next] : 0, last_next = q_first < count ? ptr[row_next + 1] : 0;
    for (int q0 = ((b - short_blocks) * (kThreads / 32) + warp) * 4; q0 < count; q0 += step) {
      const int q = q0 + grp;
      const bool have = q < count;
      const int row = row_next;
      const offset_t first = first_next, last = last_next;
      row_next = row_after;
      first_next = q + step < count ? ptr[row_next] : 0;
      last_next = q + step < count ? ptr[row_next + 1] : 0;
      row_after = q + 2 * step < count ? medium[q + 2 * step] : 0;
      const bool kept = have && (!keep_row || keep_row[row]);
      const bool grouped = have && (!kept || last - first <= kGroupRowMax);
      const offset_t end = grouped && kept ? last : first;
      const auto sides = sides_of(row);   // row 0's past the last
      // Every load of the row's (up to) four entries per lane first.
      int col[4];
      double a[4];
      double2 bnd[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const offset_t p = first + gl + 8 * j;
        col[j] = p < end ? ld_stream(idx + p, term.hint.stream) : -1;
        a[j] = p < end ? ld_stream(val + p, term.hint.stream) : 0.0;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        bnd[j] = col[j] >= 0 ? ld_keep(lu + col[j], term.hint.keep) : make_double2(0.0, 0.0);
      // Live mask over the group's 32 stored positions: bit (8j + gl) is
      // stored entry gl + 8j.
      unsigned live_mask = 0;
      bool live[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        live[j] = col[j] >= 0 && !removed_column(bnd[j]);
        live_mask |= ((__ballot_sync(0xffffffffu, live[j]) >> (grp * 8)) & 0xffu) << (8 * j);
      }
      int ni = 0, pi = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (!live[j]) continue;
        double plo, phi;
        term.slot(a[j], bnd[j], plo, phi, ni, pi);
        const int rank = __popc(live_mask & ((1u << (gl + 8 * j)) - 1u));
        glo[rank] = plo;
        ghi[rank] = phi;
      }
      __syncwarp();
      const int nlive = __popc(live_mask);
      const auto at = [&](const double* v, int r) { return r < nlive ? v[r] : 0.0; };
      double lo = (at(glo, gl) + at(glo, gl + 16)) + (at(glo, gl + 8) + at(glo, gl + 24));
      double hi = (at(ghi, gl) + at(ghi, gl + 16)) + (at(ghi, gl + 8) + at(ghi, gl + 24));
      __syncwarp();
#pragma unroll
      for (int off = 4; off > 0; off >>= 1) {
        lo = lo + __shfl_down_sync(0xffffffffu, lo, off, 8);
        hi = hi + __shfl_down_sync(0xffffffffu, hi, off, 8);
        ni = ni + __shfl_down_sync(0xffffffffu, ni, off, 8);
        pi = pi + __shfl_down_sync(0xffffffffu, pi, off, 8);
      }
      if (grouped && gl == 0) finish(row, sides, lo, hi, ni, pi);
      // Longer medium rows: one warp each, as before.
      unsigned rest = __ballot_sync(0xffffffffu, have && !grouped && gl == 0);
      while (rest) {
        const int src = __ffs(rest) - 1;
        rest &= rest - 1;
        full_row(__shfl_sync(0xffffffffu, row, src));
      }
    }
  } else {
    const int lb = b - short_blocks - medium_blocks;
    const int nlong = gridDim.x - short_blocks - medium_blocks;
    const int count = counts[1];
    for (int q = lb; q < count; q += nlong) {
      const int row = longq[q];
      const auto sides = sides_of(row);
      double lo = 0.0, hi = 0.0;
      int ni = 0, pi = 0;
      const offset_t first = ptr[row], last = ptr[row + 1];
      const bool all_live = live_deg && live_deg[row] == int(last - first);
      if (!keep_row || keep_row[row])
        live_visit_by<256>(first, last, all_live, live_at, slots, warp_counts,
                           [&](offset_t p) { term(p, term.bounds(p), lo, hi, ni, pi); });
      lo = block_sum_cub_order(lo, dagg);
      hi = block_sum_cub_order(hi, dagg);
      ni = block_sum_cub_order(ni, iagg);
      pi = block_sum_cub_order(pi, iagg);
      if (threadIdx.x == 0) finish(row, sides, lo, hi, ni, pi);
      __syncthreads();
    }
  }
  if constexpr (Plain) post_flags(test.report, found);
}

__global__ void pack_bounds_kernel(int n, const double* __restrict__ l, const double* __restrict__ u,
                                   const uint8_t* __restrict__ keep, double2* __restrict__ lu,
                                   double* __restrict__ cand_l, double* __restrict__ cand_u) {
  after_previous_kernel();
  const double removed = __longlong_as_double(static_cast<long long>(kRemovedColumnBits));
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const double lj = l[j], uj = u[j];
    lu[j] = !keep || keep[j] ? make_double2(lj, uj) : make_double2(removed, removed);
    if (cand_l) {
      cand_l[j] = lj;
      cand_u[j] = uj;
    }
  }
}

// Live degree / singleton support.  Counts and the max live position are
// order independent, so the roles follow stored length.
__device__ __forceinline__ void stats_write(int row, bool active, int count, offset_t position,
                                            const int32_t* idx, const double* val, int32_t* degree,
                                            uint8_t* empty, uint8_t* singleton, int32_t* support,
                                            double* coefficient, unsigned long long* total) {
  if (degree) degree[row] = count;
  if (empty) empty[row] = active && count == 0;
  if (singleton) singleton[row] = active && count == 1;
  if (support) support[row] = count == 1 ? idx[position] : -1;
  if (coefficient) coefficient[row] = count == 1 ? val[position] : 0.0;
  if (total && count) atomicAdd(total, (unsigned long long)count);
}

__global__ void __launch_bounds__(kThreads)
live_stats_kernel(int rows, const offset_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                  const double* __restrict__ val, const uint8_t* __restrict__ keep_outer,
                  const uint8_t* __restrict__ keep_inner, const int32_t* __restrict__ medium,
                  const int32_t* __restrict__ longq, const int32_t* __restrict__ counts, int short_blocks,
                  int medium_blocks, int32_t* degree, uint8_t* empty, uint8_t* singleton,
                  int32_t* support, double* coefficient, unsigned long long* total) {
  after_previous_kernel();
  __shared__ int scount[8];
  __shared__ long long spos[8];
  __shared__ unsigned long long stotal[8];
  const int b = blockIdx.x;
  unsigned long long acc = 0;  // live entries seen by this thread, added once per block
  if (b < short_blocks) {
    const int stride_ = short_blocks * blockDim.x;
    int r_next = b * blockDim.x + threadIdx.x;
    offset_t first_next = r_next < rows ? ptr[r_next] : 0, last_next = r_next < rows ? ptr[r_next + 1] : 0;
    for (int r = r_next; r < rows; r += stride_) {
      const offset_t first = first_next, last = last_next;
      r_next = r + stride_;   // the next row's pointers, one iteration ahead
      first_next = r_next < rows ? ptr[r_next] : 0;
      last_next = r_next < rows ? ptr[r_next + 1] : 0;
      if (last - first > kShortRow) continue;
      const bool active = !keep_outer || keep_outer[r];
      int count = 0;
      offset_t pos = -1;
      if (active)
        for (offset_t p = first; p < last; ++p)
          if (!keep_inner || keep_inner[__ldcs(idx + p)]) { ++count; pos = p; }
      stats_write(r, active, count, pos, idx, val, degree, empty, singleton, support, coefficient, nullptr);
      acc += unsigned(count);
    }
  } else if (b < short_blocks + medium_blocks) {
    // Four medium rows per warp, eight lanes each: counts and the last live
    // position are order-free, and four rows' loads are in flight at once.
    const int g = threadIdx.x & 7;
    const int nwarps = medium_blocks * (kThreads / 32);
    const int nmedium = counts[0];
    for (int q0 = ((b - short_blocks) * (kThreads / 32) + (threadIdx.x >> 5)) * 4; q0 < nmedium; q0 += nwarps * 4) {
      const int q = q0 + ((threadIdx.x & 31) >> 3);
      int r = -1, count = 0;
      bool active = false;
      long long pos = -1;
      if (q < nmedium) {
        r = medium[q];
        active = !keep_outer || keep_outer[r];
        if (active)
          for (offset_t p = ptr[r] + g; p < ptr[r + 1]; p += 8)
            if (!keep_inner || keep_inner[__ldcs(idx + p)]) { ++count; pos = p; }
      }
      for (int off = 4; off; off >>= 1) {
        count += __shfl_down_sync(0xffffffffu, count, off, 8);
        pos = max(pos, __shfl_down_sync(0xffffffffu, pos, off, 8));
      }
      if (g == 0 && r >= 0) {
        stats_write(r, active, count, offset_t(pos), idx, val, degree, empty, singleton, support, coefficient, nullptr);
        acc += unsigned(count);
      }
    }
  } else {
    const int lb = b - short_blocks - medium_blocks, nlong = gridDim.x - short_blocks - medium_blocks;
    for (int q = lb; q < counts[1]; q += nlong) {
      const int r = longq[q];
      const bool active = !keep_outer || keep_outer[r];
      int count = 0;
      long long pos = -1;
      if (active)
        for (offset_t p = ptr[r] + threadIdx.x; p < ptr[r + 1]; p += kThreads)
          if (!keep_inner || keep_inner[__ldcs(idx + p)]) { ++count; pos = p; }
      for (int off = 16; off; off >>= 1) {
        count += __shfl_down_sync(0xffffffffu, count, off);
        pos = max(pos, __shfl_down_sync(0xffffffffu, pos, off));
      }
      if ((threadIdx.x & 31) == 0) { scount[threadIdx.x >> 5] = count; spos[threadIdx.x >> 5] = pos; }
      __syncthreads();
      if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) { count += scount[w]; pos = max(pos, spos[w]); }
        stats_write(r, active, count, offset_t(pos), idx, val, degree, empty, singleton, support, coefficient, nullptr);
        acc += unsigned(count);
      }
      __syncthreads();
    }
  }
  if (!total) return;
  for (int off = 16; off; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
  if ((threadIdx.x & 31) == 0) stotal[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int w = 0; w < 8; ++w) t += stotal[w];
    if (t) atomicAdd(total, t);
  }
}

__global__ void __launch_bounds__(kThreads)
col_max_kernel(int rows, const offset_t* __restrict__ ptr, const int32_t* __restrict__ idx,
               const double* __restrict__ val, const uint8_t* __restrict__ keep_row,
               const int32_t* __restrict__ medium, const int32_t* __restrict__ longq,
               const int32_t* __restrict__ counts, int short_blocks, int medium_blocks, double* out) {
  after_previous_kernel();
  __shared__ double smax[8];
  const int b = blockIdx.x;
  if (b < short_blocks) {
    const int stride_ = short_blocks * blockDim.x;
    int r_next = b * blockDim.x + threadIdx.x;
    offset_t first_next = r_next < rows ? ptr[r_next] : 0, last_next = r_next < rows ? ptr[r_next + 1] : 0;
    for (int r = r_next; r < rows; r += stride_) {
      const offset_t first = first_next, last = last_next;
      r_next = r + stride_;   // the next row's pointers, one iteration ahead
      first_next = r_next < rows ? ptr[r_next] : 0;
      last_next = r_next < rows ? ptr[r_next + 1] : 0;
      if (last - first > kShortRow) continue;
      // All (at most 8) loads first; the max is order-free.
      int row[kShortRow];
      double a[kShortRow];
#pragma unroll
      for (int k = 0; k < kShortRow; ++k) {
        row[k] = first + k < last ? __ldcs(idx + first + k) : -1;
        a[k] = first + k < last ? __ldcs(val + first + k) : 0.0;
      }
      double v = 0.0;
#pragma unroll
      for (int k = 0; k < kShortRow; ++k)
        if (row[k] >= 0 && (!keep_row || keep_row[row[k]])) v = fmax(v, fabs(a[k]));
      out[r] = v;
    }
    return;
  }
  if (b < short_blocks + medium_blocks) {
    // Four medium rows per warp, eight lanes each (the max is order-free).
    const int g = threadIdx.x & 7;
    const int nwarps = medium_blocks * (kThreads / 32);
    const int nmedium = counts[0];
    for (int q0 = ((b - short_blocks) * (kThreads / 32) + (threadIdx.x >> 5)) * 4; q0 < nmedium; q0 += nwarps * 4) {
      const int q = q0 + ((threadIdx.x & 31) >> 3);
      int r = -1;
      double v = 0.0;
      if (q < nmedium) {
        r = medium[q];
        for (offset_t p = ptr[r] + g; p < ptr[r + 1]; p += 8)
          if (!keep_row || keep_row[__ldcs(idx + p)]) v = fmax(v, fabs(__ldcs(val + p)));
      }
      for (int off = 4; off; off >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, off, 8));
      if (g == 0 && r >= 0) out[r] = v;
    }
    return;
  }
  const int lb = b - short_blocks - medium_blocks, nlong = gridDim.x - short_blocks - medium_blocks;
  for (int q = lb; q < counts[1]; q += nlong) {
    const int r = longq[q];
    double v = 0.0;
    for (offset_t p = ptr[r] + threadIdx.x; p < ptr[r + 1]; p += kThreads)
      if (!keep_row || keep_row[idx[p]]) v = fmax(v, fabs(val[p]));
    for (int off = 16; off; off >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, off));
    if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < 8; ++w) v = fmax(v, smax[w]);
      out[r] = v;
    }
    __syncthreads();
  }
}

struct Roles {
  int short_blocks, medium_blocks, long_blocks;
};
Roles roles_for(int rows) {
  Roles r;
  r.short_blocks = grid_stride_blocks(rows, kThreads, 16);
  r.medium_blocks = std::min<int>(kNumSMs * 8, (rows + 7) / 8);
  r.long_blocks = std::min<int>(kNumSMs * 4, rows);
  return r;
}

struct ScheduleCache {
  std::array<RowSchedule, 2> slots;
  unsigned next = 0;
  uint64_t epoch = 1;
};
// Thread-lifetime caches are deliberately never destroyed: their device
// buffers live until process exit, when the driver reclaims them, so no CUDA
// call runs during thread-exit destruction (whose order relative to the
// engine stream is unspecified).
ScheduleCache& schedule_cache() {
  static thread_local ScheduleCache* c = [] {
    ctx();
    return new ScheduleCache;
  }();
  return *c;
}

}  // namespace

namespace {
// Row r writes the tiles whose first stored position, or last one (the last
// tile ends at nnz - 1), falls in [ptr[r], ptr[r+1]): every tile gets both
// rows with no search, in one pass over the row pointers.
__global__ void tile_rows_kernel(int rows, offset_t nnz, const offset_t* __restrict__ ptr, int2* __restrict__ tile_rows) {
  after_previous_kernel();
  constexpr int64_t T = kEntryTile;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
    const int64_t a = ptr[r], b = ptr[r + 1];
    if (a == b) continue;
    for (int64_t t = (a + T - 1) / T; t * T < b; ++t) tile_rows[t].x = r;
    for (int64_t t = (a + T) / T - 1; (t + 1) * T <= b; ++t) tile_rows[t].y = r;
    if (b == nnz) tile_rows[(nnz - 1) / T].y = r;
  }
}
}  // namespace

void build_schedule(RowSchedule& s, const DevCsr& M, const int32_t* live_degrees, cudaStream_t st) {
  const size_t rows = size_t(std::max(M.rows, 1));
  if (s.medium.n < rows) s.medium.alloc(rows, st);
  if (s.long_rows.n < rows) s.long_rows.alloc(rows, st);
  if (s.counts.n < 2) s.counts.alloc(2, st);
  check(cudaMemsetAsync(s.counts.p, 0, 2 * sizeof(int32_t), st), "schedule counts");
  GPP_LAUNCH(classify_rows, blocks_for(M.rows), kThreads, 0, st, M.ptr, M.rows, live_degrees, s.medium.p,
             s.long_rows.p, s.counts.p);
  s.tiles = 0;
  s.sorted = -1;
  if (!live_degrees && M.rows > 0 && M.nnz > 0) {
    s.tiles = (int64_t(M.nnz) + kEntryTile - 1) / kEntryTile;
    if (s.tile_rows.n < size_t(s.tiles)) s.tile_rows.alloc(size_t(s.tiles), st);
    GPP_LAUNCH(tile_rows_kernel, grid_stride_blocks(M.rows), kThreads, 0, st, M.rows, M.nnz, M.ptr, s.tile_rows.p);
  }
  s.ptr = M.ptr;
  s.rows = M.rows;
  s.nnz = M.nnz;
  s.epoch = live_degrees ? 0 : schedule_cache().epoch;
}

const RowSchedule& stored_schedule(const DevCsr& M) {
  auto& c = schedule_cache();
  for (auto& s : c.slots)
    if (s.epoch == c.epoch && s.ptr == M.ptr && s.rows == M.rows && s.nnz == M.nnz) return s;
  auto& s = c.slots[c.next++ % c.slots.size()];
  build_schedule(s, M, nullptr, ctx().stream);
  return s;
}

void invalidate_schedules() { ++schedule_cache().epoch; }

void forget_schedule(const offset_t* ptr) {
  if (!ptr) return;
  for (auto& s : schedule_cache().slots)
    if (s.ptr == ptr) s.ptr = nullptr;
}

void live_stats_side(const DevCsr& M, const uint8_t* keep_outer, const uint8_t* keep_inner, int32_t* degree,
                     uint8_t* empty, uint8_t* singleton, int32_t* support, double* coefficient,
                     unsigned long long* total, cudaStream_t s) {
  if (!M.rows) return;
  const RowSchedule& sch = stored_schedule(M);
  const Roles r = roles_for(M.rows);
  // Algorithmic bytes: row pointers, inner indices, both masks, five outputs.
  const double bytes = 4.0 * (M.rows + 1) + 4.0 * M.nnz + (keep_outer ? M.rows : 0) + (keep_inner ? M.cols : 0) +
                       double(M.rows) * ((degree ? 4 : 0) + (empty ? 1 : 0) + (singleton ? 1 : 0) +
                                         (support ? 4 : 0) + (coefficient ? 8 : 0));
  GPP_LAUNCH_BYTES(live_stats_kernel, bytes, r.short_blocks + r.medium_blocks + r.long_blocks, kThreads, 0, s, M.rows,
             M.ptr, M.idx, M.val, keep_outer, keep_inner, sch.medium.p, sch.long_rows.p, sch.counts.p,
             r.short_blocks, r.medium_blocks, degree, empty, singleton, support, coefficient, total);
}

void allocate_stats(Stats& st, int32_t m, int32_t n) {
  auto s = ctx().stream;
  st.row_nnz.alloc(size_t(m), s); st.empty_row.alloc(size_t(m), s); st.singleton_row.alloc(size_t(m), s);
  st.srow_col.alloc(size_t(m), s); st.srow_val.alloc(size_t(m), s);
  st.col_nnz.alloc(size_t(n), s); st.empty_col.alloc(size_t(n), s); st.singleton_col.alloc(size_t(n), s);
  st.scol_row.alloc(size_t(n), s); st.scol_val.alloc(size_t(n), s);
  st.live_nnz.alloc(1, s);
  st.seen_row.alloc(size_t(m), s); st.seen_col.alloc(size_t(n), s);
  st.dirty_row.alloc(size_t(m), s); st.dirty_col.alloc(size_t(n), s);
  st.deleted.alloc(size_t(m) + size_t(n), s);
  st.counters.alloc(2, s);
  st.valid = false;
}

namespace {

// ---- incremental refresh ---------------------------------------------------
//
// Masks only lose entries between two materialisations, so the statistics of
// the current masks follow from those of the previous ones: a deleted row
// takes one off the degree of every still-kept column it touches (and a
// deleted column likewise for rows), the live total drops by the entries that
// stopped being live, and only rows / columns whose degree changed need their
// empty / singleton flags and singleton support recomputed.  The result is
// the full recount's exactly (integer counts, and the support of a degree-1
// row is its only live entry).

// Items of one mask that went from kept to deleted, appended to `list`; the
// mask last seen is brought up to date.  Sixteen mask bytes per thread: between
// two refreshes almost no byte differs, so a sweep costs two bytes read and
// one written per item.
__device__ __forceinline__ void find_deleted(int n, uint8_t* __restrict__ seen, const uint8_t* __restrict__ keep,
                                             int32_t* __restrict__ list, int32_t* counter) {
  const int lane = threadIdx.x & 31;
  const int chunks = (n + 15) / 16;
  const int stride = gridDim.x * blockDim.x;
  const int top = (chunks + stride - 1) / stride * stride;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < top; c += stride) {
    unsigned gone = 0;   // bit q: item 16 c + q
    const int base = c * 16;
    if (base + 16 <= n) {
      const uint4 a = reinterpret_cast<const uint4*>(seen)[c], b = reinterpret_cast<const uint4*>(keep)[c];
      if (a.x != b.x || a.y != b.y || a.z != b.z || a.w != b.w) {
        for (int q = 0; q < 16; ++q)
          if (seen[base + q] && !keep[base + q]) gone |= 1u << q;
        reinterpret_cast<uint4*>(seen)[c] = b;
      }
    } else {
      for (int q = 0; q < 16 && base + q < n; ++q) {
        if (seen[base + q] && !keep[base + q]) gone |= 1u << q;
        seen[base + q] = keep[base + q];
      }
    }
    if (!__any_sync(0xffffffffu, gone != 0)) continue;
    const int mine = __popc(gone);
    int incl = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int peer = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += peer;
    }
    int at = 0;
    if (lane == 31) at = atomicAdd(counter, incl);
    at = __shfl_sync(0xffffffffu, at, 31) + incl - mine;
    for (unsigned g = gone; g; g &= g - 1) list[at++] = base + __ffs(g) - 1;
  }
}
// Deleted rows to list[0 ..], deleted columns to list[m ..]; `counters` holds
// their numbers (zero at launch).
__global__ void inc_deleted(int m, int n, uint8_t* __restrict__ seen_row, const uint8_t* __restrict__ keep_row,
                            uint8_t* __restrict__ seen_col, const uint8_t* __restrict__ keep_col,
                            int32_t* __restrict__ list, int32_t* counters) {
  after_previous_kernel();
  find_deleted(m, seen_row, keep_row, list, counters);
  find_deleted(n, seen_col, keep_col, list + m, counters + 1);
}

// One side's arrays of the statistics.
struct SideStats {
  const offset_t* ptr;
  const int32_t* idx;
  const double* val;
  const uint8_t* keep;
  int32_t* degree;
  uint8_t *empty, *singleton;
  int32_t* support;
  double* coefficient;
  uint8_t* dirty;
};

// Still-kept items among entries p, p + step, .. of a deleted one: each loses one
// degree and is marked dirty.  Returns their number.
__device__ __forceinline__ int leave_inner(const SideStats& outer, const SideStats& inner, int64_t p, offset_t end,
                                           int step) {
  int left = 0;
  for (; p < end; p += 4 * step) {
    int c[4];
    bool kept[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) c[k] = end - p > k * step ? outer.idx[p + k * step] : -1;
#pragma unroll
    for (int k = 0; k < 4; ++k) kept[k] = c[k] >= 0 && inner.keep[c[k]];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (!kept[k]) continue;
      atomicSub(inner.degree + c[k], 1);
      inner.dirty[c[k]] = 1;
      ++left;
    }
  }
  return left;
}
// Deleted rows by the first half of the blocks, deleted columns by the rest
// (the halves touch different items: a deleted item's own statistics, and the
// degrees of kept items of the other side).  Eight lanes per deleted item, four items
// to a warp, taken so that few items go to warps of their own; one of more than
// kWideItem entries by its whole warp.  A deleted item's own statistics are reset, and
// every still-kept item it touches loses one degree and is marked dirty.  The live total
// drops by a deleted row's old degree and, for a deleted column, by one per kept row it
// leaves; added up in registers, one atomic per warp (an atomic per item on the one total
// took 152 us when 0.8M rows went at once, on the QAP N = 30 relaxation).  Bound by the
// round trips of an item's entries: eight lanes to the 4 rows of 400,000 entries of a
// 200,000 x 500,000 LP took 19.0 ms, a warp with one entry a lane in flight 6.6 ms, this
// 2.8 ms.
constexpr int kWideItem = 64;
__device__ __forceinline__ void walk_deleted(int m, const int32_t* list, const int32_t* counters,
                                             const SideStats& rows, const SideStats& cols,
                                             unsigned long long* live_nnz) {
  const int half = gridDim.x / 2;
  const bool row_side = int(blockIdx.x) < half;
  const SideStats& outer = row_side ? rows : cols;
  const SideStats& inner = row_side ? cols : rows;
  const int32_t* deleted = row_side ? list : list + m;
  const int count = counters[row_side ? 0 : 1];
  const int lane = threadIdx.x & 31, gl = lane & 7;
  const int block = row_side ? int(blockIdx.x) : int(blockIdx.x) - half;
  const int64_t warps = int64_t(row_side ? half : int(gridDim.x) - half) * (kThreads / 32);
  unsigned long long dropped = 0;
  for (int64_t w0 = block * (kThreads / 32) + (threadIdx.x >> 5); w0 < count; w0 += warps * 4) {
    const int64_t w = w0 + (lane >> 3) * warps;
    const bool have = w < count;
    const int r = have ? deleted[w] : 0;
    const offset_t first = have ? outer.ptr[r] : 0, end = have ? outer.ptr[r + 1] : 0;
    const bool wide = end - first > kWideItem;
    int left = wide ? 0 : leave_inner(outer, inner, int64_t(first) + gl, end, 8);
    for (unsigned rest = __ballot_sync(0xffffffffu, wide && gl == 0); rest; rest &= rest - 1) {
      const int src = __ffs(rest) - 1;
      const offset_t f = __shfl_sync(0xffffffffu, first, src), e = __shfl_sync(0xffffffffu, end, src);
      left += leave_inner(outer, inner, int64_t(f) + lane, e, 32);
    }
    if (!row_side) dropped += unsigned(left);
    if (have && gl == 0) {
      if (row_side) dropped += (unsigned long long)outer.degree[r];
      outer.degree[r] = 0; outer.empty[r] = 0; outer.singleton[r] = 0; outer.support[r] = -1;
      outer.coefficient[r] = 0.0;
    }
  }
  for (int off = 16; off; off >>= 1) dropped += __shfl_down_sync(0xffffffffu, dropped, off);
  if (lane == 0 && dropped) atomicAdd(live_nnz, 0ULL - dropped);
}
__global__ void __launch_bounds__(kThreads) inc_walk(int m, const int32_t* list, const int32_t* counters,
                                                     SideStats rows, SideStats cols, unsigned long long* live_nnz) {
  after_previous_kernel();
  walk_deleted(m, list, counters, rows, cols, live_nnz);
}

// Flags of the dirty kept items; a degree-1 item finds its only live entry.
// Four items per thread (most dirty bytes are clear).
__device__ __forceinline__ void fix_dirty(int n, const SideStats& outer, const uint8_t* __restrict__ keep_inner) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c * 4 < n; c += gridDim.x * blockDim.x) {
    const int base = c * 4;
    if (base + 4 <= n && reinterpret_cast<const uint32_t*>(outer.dirty)[c] == 0) continue;
    for (int r = base; r < base + 4 && r < n; ++r) {
      if (!outer.dirty[r]) continue;
      outer.dirty[r] = 0;
      if (!outer.keep[r]) continue;
      const int d = outer.degree[r];
      outer.empty[r] = d == 0;
      outer.singleton[r] = d == 1;
      int sup = -1;
      double coef = 0.0;
      if (d == 1)
        for (offset_t p = outer.ptr[r]; p < outer.ptr[r + 1]; ++p)
          if (keep_inner[outer.idx[p]]) { sup = outer.idx[p]; coef = outer.val[p]; }
      outer.support[r] = sup;
      outer.coefficient[r] = coef;
    }
  }
}
__global__ void inc_fix(int m, int n, SideStats rows, SideStats cols, int32_t* __restrict__ counters,
                        const unsigned long long* __restrict__ live_nnz, Mailbox* box, uint32_t seq) {
  after_previous_kernel();
  if (blockIdx.x == 0 && threadIdx.x < 2) counters[threadIdx.x] = 0;   // for the next refresh
  if (blockIdx.x == 0 && threadIdx.x == 0) post_values(box, seq, int64_t(*live_nnz));
  fix_dirty(m, rows, cols.keep);
  fix_dirty(n, cols, rows.keep);
}

// The three in one cluster, for small models.
__global__ void __cluster_dims__(kSmallCluster, 1, 1) __launch_bounds__(kThreads)
inc_small(int m, int n, uint8_t* seen_row, uint8_t* seen_col, int32_t* list, int32_t* counters, SideStats rows,
          SideStats cols, unsigned long long* live_nnz, Mailbox* box, uint32_t seq) {
  after_previous_kernel();
  find_deleted(m, seen_row, rows.keep, list, counters);
  find_deleted(n, seen_col, cols.keep, list + m, counters + 1);
  cluster_barrier();
  walk_deleted(m, list, counters, rows, cols, live_nnz);
  cluster_barrier();
  if (blockIdx.x == 0 && threadIdx.x < 2) counters[threadIdx.x] = 0;   // for the next refresh
  if (blockIdx.x == 0 && threadIdx.x == 0)
    post_values(box, seq, int64_t(*static_cast<volatile unsigned long long*>(live_nnz)));
  fix_dirty(m, rows, cols.keep);
  fix_dirty(n, cols, rows.keep);
}

// Statistics of a model all of whose rows and columns are kept: the degrees
// are the stored lengths, so nothing but the row pointers (and a one-entry
// item's entry) is read.
__device__ __forceinline__ void full_item(int r, const SideStats& s, uint8_t* __restrict__ seen) {
  const offset_t first = s.ptr[r];
  const int d = int(s.ptr[r + 1] - first);
  s.degree[r] = d;
  s.empty[r] = d == 0;
  s.singleton[r] = d == 1;
  s.support[r] = d == 1 ? s.idx[first] : -1;
  s.coefficient[r] = d == 1 ? s.val[first] : 0.0;
  s.dirty[r] = 0;
  seen[r] = 1;
}
__global__ void stats_of_full_model(int m, int n, offset_t nnz, SideStats rows, SideStats cols,
                                    uint8_t* __restrict__ seen_row, uint8_t* __restrict__ seen_col,
                                    unsigned long long* __restrict__ live_nnz, int32_t* __restrict__ counters) {
  after_previous_kernel();
  const int top = n > m ? n : m;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < top; k += gridDim.x * blockDim.x) {
    if (k == 0) {
      *live_nnz = (unsigned long long)nnz;
      counters[0] = counters[1] = 0;
    }
    if (k < m) full_item(k, rows, seen_row);
    if (k < n) full_item(k, cols, seen_col);
  }
}

}  // namespace

void refresh_stats(Stats& st, const WorkingLp& lp, const Plan& plan) {
  // refresh_live_stats (gpu_presolve_kernels.cu:493-517).
  auto s = ctx().stream;
  const int m = lp.m(), n = lp.n();
  const SideStats rows{lp.A.ptr, lp.A.idx, lp.A.val, plan.keep_row.p, st.row_nnz.p, st.empty_row.p, st.singleton_row.p,
                       st.srow_col.p, st.srow_val.p, st.dirty_row.p};
  const SideStats cols{lp.AT.ptr, lp.AT.idx, lp.AT.val, plan.keep_col.p, st.col_nnz.p, st.empty_col.p,
                       st.singleton_col.p, st.scol_row.p, st.scol_val.p, st.dirty_col.p};
  if (!st.valid && plan.all_kept && std::max(m, n) > 0) {
    // A full recount normally follows a fresh plan, whose masks keep every
    // row and column (the host knows: Plan::all_kept).
    GPP_LAUNCH_BYTES(stats_of_full_model, 22.0 * (double(m) + n), grid_stride_blocks(std::max(m, n)), kThreads, 0, s, m,
                     n, lp.A.nnz, rows, cols, st.seen_row.p, st.seen_col.p, st.live_nnz.p, st.counters.p);
    st.nnz_known = lp.A.nnz;
  } else if (!st.valid) {
    st.live_nnz.zero();
    st.dirty_row.zero();
    st.dirty_col.zero();
    st.counters.zero();
    live_stats_side(lp.A, plan.keep_row.p, plan.keep_col.p, st.row_nnz.p, st.empty_row.p, st.singleton_row.p,
                    st.srow_col.p, st.srow_val.p, st.live_nnz.p, s);
    live_stats_side(lp.AT, plan.keep_col.p, plan.keep_row.p, st.col_nnz.p, st.empty_col.p, st.singleton_col.p,
                    st.scol_row.p, st.scol_val.p, nullptr, s);
    st.seen_row.copy_from(plan.keep_row.p, size_t(m));
    st.seen_col.copy_from(plan.keep_col.p, size_t(n));
    st.nnz_known = int64_t(read_scalar(st.live_nnz.p));
  } else {
    const uint32_t seq = ++ctx().nnz_seq;
    Mailbox* const box = ctx().nnz_box(seq);
    if (small_model(m, n, lp.A.nnz)) {
      GPP_LAUNCH_BYTES(inc_small, 2.0 * (double(m) + n), kSmallCluster, kThreads, 0, s, m, n, st.seen_row.p,
                       st.seen_col.p, st.deleted.p, st.counters.p, rows, cols, st.live_nnz.p, box, seq);
    } else {
      GPP_LAUNCH_BYTES(inc_deleted, 2.0 * (double(m) + n), grid_stride_blocks(std::max(m, n) / 16 + 1), kThreads, 0, s,
                       m, n, st.seen_row.p, plan.keep_row.p, st.seen_col.p, plan.keep_col.p, st.deleted.p,
                       st.counters.p);
      const int g = 2 * std::max(1, std::min(kNumSMs * 4, (std::max(m, n) + kThreads / 8 - 1) / (kThreads / 8)));
      GPP_LAUNCH(inc_walk, g, kThreads, 0, s, m, st.deleted.p, st.counters.p, rows, cols, st.live_nnz.p);
      GPP_LAUNCH(inc_fix, grid_stride_blocks(std::max(m, n) / 4 + 1), kThreads, 0, s, m, n, rows, cols, st.counters.p,
                 st.live_nnz.p, box, seq);
    }
    st.nnz_known = -1;
    st.nnz_seq = seq;
  }
  static std::atomic<uint64_t> versions{0};
  st.version = ++versions;
  st.valid = true;
}

void pack_bounds(const double* l, const double* u, const uint8_t* keep_col, int32_t n, double2* lu,
                 cudaStream_t s, double* cand_l, double* cand_u) {
  if (n <= 0) return;
  GPP_LAUNCH_BYTES(pack_bounds_kernel, (cand_l ? 49.0 : 33.0) * n, grid_stride_blocks(n), kThreads, 0, s, n, l, u,
                   keep_col, lu, cand_l, cand_u);
}

namespace {
template <Sums Form>
void launch_activity(const DevCsr& A, const double2* lu, double zero_tol, const uint8_t* keep_row,
                     const int32_t* live_deg, double* lo, double* hi, int32_t* ni, int32_t* pi, double out_bytes,
                     cudaStream_t s, uint64_t degrees_version, const RedundantTest& test = {},
                     const RowRecords& records = {}) {
  static thread_local RowSchedule* live_schedule = new RowSchedule;  // never destroyed (see schedule_cache)
  const RowSchedule* sch;
  if (live_deg) {
    // Statistics versions are unique in the process, so one names its matrix
    // and degrees; callers with degrees of their own give 0.
    if (degrees_version == 0 || live_schedule->degrees_version != degrees_version) {
      build_schedule(*live_schedule, A, live_deg, s);
      live_schedule->degrees_version = degrees_version;
    }
    sch = live_schedule;
  } else {
    sch = &stored_schedule(A);
  }
  const Roles r = roles_for(A.rows);
  // Algorithmic bytes (each array charged once): row pointers, column indices
  // and values, packed column bounds, row mask, live degrees, the outputs.
  const double bytes = 4.0 * (A.rows + 1) + 12.0 * A.nnz + 16.0 * A.cols + (keep_row ? A.rows : 0) +
                       (live_deg ? 4.0 * A.rows : 0) + out_bytes * A.rows;
  const int grid = r.short_blocks + r.medium_blocks + r.long_blocks;
  if constexpr (Form == Sums::kPlain)
    GPP_LAUNCH_BYTES(activity_kernel<Sums::kPlain>, bytes, grid, kThreads, 0, s, A.rows, A.ptr, A.idx, A.val, lu,
                     zero_tol, keep_row, live_deg, sch->medium.p, sch->long_rows.p, sch->counts.p, r.short_blocks,
                     r.medium_blocks, lo, hi, ni, pi, records, test);
  else if constexpr (Form == Sums::kRecords)
    GPP_LAUNCH_BYTES(activity_kernel<Sums::kRecords>, bytes, grid, kThreads, 0, s, A.rows, A.ptr, A.idx, A.val, lu,
                     zero_tol, keep_row, live_deg, sch->medium.p, sch->long_rows.p, sch->counts.p, r.short_blocks,
                     r.medium_blocks, lo, hi, ni, pi, records, test);
  else
    GPP_LAUNCH_BYTES(activity_kernel<Sums::kFinite>, bytes, grid, kThreads, 0, s, A.rows, A.ptr, A.idx, A.val, lu,
                     zero_tol, keep_row, live_deg, sch->medium.p, sch->long_rows.p, sch->counts.p, r.short_blocks,
                     r.medium_blocks, lo, hi, ni, pi, records, test);
}
}  // namespace

void row_activity_summary_packed(const DevCsr& A, const double2* lu, double zero_tol, const uint8_t* keep_row,
                                 const int32_t* live_deg, double* min_fin, double* max_fin, int32_t* min_inf,
                                 int32_t* max_inf, cudaStream_t s, uint64_t degrees_version) {
  // compute_row_activity_summary (gpu_presolve_kernels.cu:744-787).
  if (!A.rows) return;
  launch_activity<Sums::kFinite>(A, lu, zero_tol, keep_row, live_deg, min_fin, max_fin, min_inf, max_inf, 24.0, s,
                         degrees_version);
}

void row_activity_summary(const DevCsr& A, const double* l, const double* u, double zero_tol,
                          const uint8_t* keep_row, const uint8_t* keep_col, const int32_t* live_deg,
                          double* min_fin, double* max_fin, int32_t* min_inf, int32_t* max_inf,
                          cudaStream_t s) {
  if (!A.rows) return;
  DBuf<double2> lu(size_t(std::max(A.cols, 1)), s);
  pack_bounds(l, u, keep_col, A.cols, lu.p, s);
  row_activity_summary_packed(A, lu.p, zero_tol, keep_row, live_deg, min_fin, max_fin, min_inf, max_inf, s);
}

void row_activity_records(const DevCsr& A, const double2* lu, double zero_tol, const Plan& plan,
                          const int32_t* live_deg, const RowRecords& out, cudaStream_t s, uint64_t degrees_version) {
  if (!A.rows) return;
  RedundantTest sides{};
  sides.AL = plan.AL.p;
  sides.AU = plan.AU.p;
  launch_activity<Sums::kRecords>(A, lu, zero_tol, plan.keep_row.p, live_deg, nullptr, nullptr, nullptr, nullptr, 49.0,
                                  s, degrees_version, sides, out);
}

void redundant_rows_test(const DevCsr& A, const double2* lu, const uint8_t* keep_row, const int32_t* live_deg,
                         const RedundantTest& test, cudaStream_t s, uint64_t degrees_version) {
  launch_activity<Sums::kPlain>(A, lu, 0.0, keep_row, live_deg, nullptr, nullptr, nullptr, nullptr, 17.0, s, degrees_version,
                        test);
}

void mirror_bounds(Plan& plan, int32_t n, cudaStream_t s) {
  if (plan.bounds_mirrored) return;
  if (plan.lu.n < size_t(n)) {
    plan.lu.alloc(size_t(n), s);
    plan.cand_l.alloc(size_t(n), s);
    plan.cand_u.alloc(size_t(n), s);
  }
  pack_bounds(plan.l.p, plan.u.p, plan.keep_col.p, n, plan.lu.p, s, plan.cand_l.p, plan.cand_u.p);
  plan.bounds_mirrored = true;
}

void col_max_abs(const DevCsr& AT, const uint8_t* keep_row, double* out, cudaStream_t s) {
  // compute_col_max_abs (gpu_presolve_kernels.cu:789-809).
  if (!AT.rows) return;
  const RowSchedule& sch = stored_schedule(AT);
  const Roles r = roles_for(AT.rows);
  const double bytes = 4.0 * (AT.rows + 1) + 12.0 * AT.nnz + (keep_row ? AT.cols : 0) + 8.0 * AT.rows;
  GPP_LAUNCH_BYTES(col_max_kernel, bytes, r.short_blocks + r.medium_blocks + r.long_blocks, kThreads, 0, s, AT.rows,
             AT.ptr, AT.idx, AT.val, keep_row, sch.medium.p, sch.long_rows.p, sch.counts.p, r.short_blocks,
             r.medium_blocks, out);
}

}  // namespace gpp

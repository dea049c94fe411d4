// The presolve scheduler: a fixed-point loop of Cleanup, Propagation,
// Aggregation and Parallel phases over a deferred plan that is materialised
// (compacted) at phase boundaries.
//
// Reference: run_gpu_presolve_impl (cpp/src/presolve/gpu_presolve.cu:2081-2645),
// apply_plan_to_working_lp (:1953-2072), capture_cleanup_recovery
// (device_recovery.cu:1011-1027).  The phase machine, the iteration budget,
// the bound-only round limit and the nnz-progress tests follow the reference
// step for step; every rule reports through one status readback.
#include <chrono>
#include <cmath>
#include <tuple>

#include "engine.cuh"
#include "presolve.hpp"

namespace gpp {

void WorkingLp::free_owned() {
  if (!owns) return;
  free_csr(A);
  free_csr(AT);
  dfree(c); dfree(AL); dfree(AU); dfree(l); dfree(u);
  c = AL = AU = l = u = nullptr;
  owns = false;
}

namespace {

// A model's vectors: columns' c, l, u and rows' AL, AU.
struct Vectors {
  double *c, *l, *u, *AL, *AU;
};

__device__ __forceinline__ void copy_at(int k, int m, int n, const Vectors& from, const Vectors& to) {
  if (k < n) {
    to.c[k] = from.c[k];
    to.l[k] = from.l[k];
    to.u[k] = from.u[k];
  }
  if (k < m) {
    to.AL[k] = from.AL[k];
    to.AU[k] = from.AU[k];
  }
}
__global__ void copy_vectors(int m, int n, Vectors from, Vectors to) {
  after_previous_kernel();
  const int top = n > m ? n : m;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < top; k += gridDim.x * blockDim.x) copy_at(k, m, n, from, to);
}

// A fresh plan in one launch: all rows and columns kept, the vectors copied.
__global__ void fresh_plan(int m, int n, Vectors from, Vectors to, uint8_t* __restrict__ keep_row,
                           uint8_t* __restrict__ keep_col) {
  after_previous_kernel();
  const int top = n > m ? n : m;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < top; k += gridDim.x * blockDim.x) {
    if (k < n) keep_col[k] = 1;
    if (k < m) keep_row[k] = 1;
    copy_at(k, m, n, from, to);
  }
}

// The kept rows' and columns' vectors and original ids to their new places,
// one launch for all of them.
__global__ void gather_kept(int m, int n, const int32_t* __restrict__ rmap, const int32_t* __restrict__ cmap,
                            Vectors from, Vectors to, const int32_t* __restrict__ rows, int32_t* __restrict__ rows_to,
                            const int32_t* __restrict__ cols, int32_t* __restrict__ cols_to) {
  after_previous_kernel();
  const int top = n > m ? n : m;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < top; k += gridDim.x * blockDim.x) {
    if (k < n) {
      const int j = cmap[k];
      if (j >= 0) {
        to.c[j] = from.c[k];
        to.l[j] = from.l[k];
        to.u[j] = from.u[k];
        if (cols_to) cols_to[j] = cols[k];
      }
    }
    if (k < m) {
      const int i = rmap[k];
      if (i >= 0) {
        to.AL[i] = from.AL[k];
        to.AU[i] = from.AU[k];
        if (rows_to) rows_to[i] = rows[k];
      }
    }
  }
}

struct Engine {
  const gpp_params& p;
  PresolveOutput& out;
  WorkingLp cur;
  bool terminal = false;
  bool active = false, pending = false;
  bool reshaped = false;   // a rule since the plan's start acted on rows or columns
  bool unsaved = false;    // the plan's vectors are ahead of the working LP's
  Plan plan;
  Stats stats;
  bool stats_dirty = true;
  uint32_t* inf_hist = nullptr;   // histogram features (scheduled runs only)
  uint64_t deletion_serial = 0;

  Engine(const gpp_params& params, PresolveOutput& o) : p(params), out(o) {}

  cudaStream_t s() const { return ctx().stream; }
  static Vectors vectors(const WorkingLp& lp) { return {lp.c, lp.l, lp.u, lp.AL, lp.AU}; }
  static Vectors vectors(const Plan& pl) { return {pl.c.p, pl.l.p, pl.u.p, pl.AL.p, pl.AU.p}; }

  void init_plan(Plan& pl) {
    const int m = cur.m(), n = cur.n();
    pl.keep_row.alloc(size_t(m), s());
    pl.keep_col.alloc(size_t(n), s());
    pl.c.alloc(size_t(n), s());
    pl.l.alloc(size_t(n), s());
    pl.u.alloc(size_t(n), s());
    pl.AL.alloc(size_t(m), s());
    pl.AU.alloc(size_t(m), s());
    GPP_LAUNCH_BYTES(fresh_plan, 49.0 * n + 33.0 * m, grid_stride_blocks(std::max(m, n)), kThreads, 0, s(), m, n,
                     vectors(cur), vectors(pl), pl.keep_row.p, pl.keep_col.p);
    pl.all_kept = true;
  }
  void prepare() {
    if (active) return;
    plan = Plan{};
    init_plan(plan);
    plan.inf_hist = inf_hist;
    plan.save_committed = [this] {
      if (!pending) save_vectors();
    };
    allocate_stats(stats, cur.m(), cur.n());
    stats_dirty = true;
    active = true;
    reshaped = false;
  }
  void refresh() {
    if (stats_dirty) {
      refresh_stats(stats, cur, plan);
      stats_dirty = false;
    }
  }
  // The live nnz of the plan as it stands.  A refresh posts it to the host, so
  // it can be asked for when it is needed: the count before a phase is used
  // only by the progress test after it, when it has long arrived.
  struct LaterCount {
    int64_t known = -1;
    uint32_t seq = 0;
  };
  LaterCount live_nnz_later() {
    if (!active) return {cur.A.nnz, 0};
    refresh();
    return {stats.nnz_known, stats.nnz_seq};
  }
  int64_t value(const LaterCount& c) const {
    return c.known >= 0 ? c.known : ctx().await(ctx().nnz_box(c.seq), c.seq, "live nnz")[0];
  }
  int64_t live_nnz() { return value(live_nnz_later()); }

  template <class F>
  bool deferred_rule(bool enabled, const char* name, F rule) {
    if (!enabled || terminal) return false;
    const NvtxRange range(name);
    prepare();
    refresh();
    // The statistics are fresh, so the column mask they describe is the
    // rule's entry mask; it stays as it is until the next refresh.
    plan.rule_entry_keep_col = stats.seen_col.p;
    plan.has_change = plan.has_row_action = plan.has_col_action = false;
    plan.has_redundant_row_deletion = plan.has_row_deletion = false;
    plan.obj_delta = 0.0;
    plan.all_kept = false;
    rule();
    out.has_infeasible = plan.has_infeasible;
    out.has_unbounded = plan.has_unbounded;
    terminal = plan.has_infeasible || plan.has_unbounded;
    const bool changed = plan.has_change && !terminal;
    if (changed) {
      if (plan.has_row_deletion || plan.has_col_action) ++deletion_serial;
      cur.obj.add(plan.obj_delta);
      capture_tape(out.record, plan.tape);
      if (plan.has_col_action)
        append_fixed(out.record, plan.keep_col.p, stats.seen_col.p, plan.l.p, plan.u.p, cur.n());
      pending = true;
      if (plan.has_row_action || plan.has_col_action) stats_dirty = reshaped = true;
      if (plan.has_col_action) plan.bounds_mirrored = false;
    } else {
      plan.tape.clear();
    }
    plan.obj_delta = 0.0;
    out.trace.push_back(std::string("rule=") + name + " changed=" + (changed ? "1" : "0"));
    return changed;
  }

  // A rule that a probe of the unchanged plan showed would change nothing:
  // the bookkeeping deferred_rule does for an unchanged rule, without
  // running it.
  bool skipped_rule(bool enabled, const char* name) {
    if (!enabled || terminal) return false;
    prepare();
    refresh();
    out.trace.push_back(std::string("rule=") + name + " changed=0");
    return false;
  }

  // apply_plan_to_working_lp (gpu_presolve.cu:1953-2072).
  void apply(Plan& pl, bool cleanup_captured) {
    const NvtxRange range("materialize");
    Record& r = out.record;
    const int m = cur.m(), n = cur.n();
    // The old -> new maps' kept counts also tell whether the plan removes
    // anything (one readback for both questions).
    DBuf<int32_t> rmap(size_t(std::max(m, 1)), s()), cmap(size_t(std::max(n, 1)), s());
    const auto [m_new, n_new] = build_old_to_new_pair(pl.keep_row.p, m, rmap.p, pl.keep_col.p, n, cmap.p, s());
    if (cur.owns && !pl.has_new_A && m_new == m && n_new == n) {
      capture_tape(r, pl.tape);
      GPP_LAUNCH_BYTES(gather_kept, 52.0 * n + 36.0 * m, grid_stride_blocks(std::max(m, n)), kThreads, 0, s(), m, n,
                       rmap.p, cmap.p, vectors(pl), vectors(cur), nullptr, nullptr, nullptr, nullptr);
      cur.obj.add(pl.obj_delta);
      return;
    }
    WorkingLp next;
    if (pl.has_new_A) {
      next.A = compact_csr(pl.new_A, rmap.p, m_new, cmap.p, n_new, s());
      next.AT = transpose_csr(next.A, s());
    } else if (cur.AT_sorted()) {
      std::tie(next.A, next.AT) = compact_csr_pair(cur.A, cur.AT, rmap.p, m_new, cmap.p, n_new, s());
      if (next.A.nnz != next.AT.nnz) throw std::logic_error("compaction: A and A^T kept different entry counts");
      next.a_sorted = cur.a_sorted;
    } else {
      next.A = compact_csr(cur.A, rmap.p, m_new, cmap.p, n_new, s());
      next.AT = transpose_csr(next.A, s());
      next.a_sorted = cur.a_sorted;
    }
    next.at_sorted = 1;
    next.c = dalloc<double>(size_t(n_new));
    next.l = dalloc<double>(size_t(n_new));
    next.u = dalloc<double>(size_t(n_new));
    next.AL = dalloc<double>(size_t(m_new));
    next.AU = dalloc<double>(size_t(m_new));
    next.obj = cur.obj;
    next.obj.add(pl.obj_delta);
    // update_device_recovery (device_recovery.cu:892-975).
    capture_tape(r, pl.tape);
    if (pl.absval) {
      capture_absolute_value(r, std::move(*pl.absval));
      pl.absval.reset();
    }
    if (pl.varpair) {
      capture_variable_pair(r, std::move(*pl.varpair));
      pl.varpair.reset();
    }
    if (!cleanup_captured && n_new != n) append_fixed(r, pl.keep_col.p, nullptr, pl.l.p, pl.u.p, n);
    globalize_segments(r);
    // The vectors and, where the maps change, the original ids.
    DBuf<int32_t> rows, cols;
    if (m_new != r.m) rows.alloc(size_t(m_new), s());
    if (n_new != r.n) cols.alloc(size_t(n_new), s());
    GPP_LAUNCH_BYTES(gather_kept, 28.0 * n + 20.0 * m + 28.0 * n_new + 20.0 * m_new, grid_stride_blocks(std::max(m, n)),
                     kThreads, 0, s(), m, n, rmap.p, cmap.p, vectors(pl), vectors(next), r.rows.p, rows.p, r.cols.p,
                     cols.p);
    if (m_new != r.m) {
      r.rows = std::move(rows);
      r.m = m_new;
    }
    if (n_new != r.n) {
      r.cols = std::move(cols);
      r.n = n_new;
    }
    cur.free_owned();
    next.owns = true;
    cur = next;
    invalidate_schedules();
  }

  // The open plan's vectors to the working LP (nothing else differs).
  void save_vectors() {
    if (!unsaved) return;
    const int m = cur.m(), n = cur.n();
    GPP_LAUNCH_BYTES(copy_vectors, 48.0 * n + 32.0 * m, grid_stride_blocks(std::max(m, n)), kThreads, 0, s(), m, n,
                     vectors(plan), vectors(cur));
    unsaved = false;
  }

  void materialize(const char* boundary) {
    // Most propagation rounds move a few bounds and nothing else: then the
    // plan, whose masks still keep everything, its statistics and its row
    // queues serve the next phase as they are; the vectors reach the working
    // LP when something reads them there.  A plan without a change stays open
    // too.
    if (active && !reshaped && (!pending || cur.owns)) {
      if (pending) out.trace.push_back(std::string("apply=") + boundary);
      unsaved = unsaved || pending;
      pending = false;
      return;
    }
    if (active && pending) {
      apply(plan, true);
      out.trace.push_back(std::string("apply=") + boundary);
    } else if (active) {
      save_vectors();
    }
    unsaved = false;
    active = pending = reshaped = false;
    plan = Plan{};
    stats = Stats{};
  }

  template <class F>
  bool materialized_rule(bool enabled, const char* name, F rule) {
    if (!enabled || terminal) return false;
    const NvtxRange range(name);
    save_vectors();
    Plan pl;
    init_plan(pl);
    rule(pl);
    out.has_infeasible = pl.has_infeasible;
    out.has_unbounded = pl.has_unbounded;
    terminal = pl.has_infeasible || pl.has_unbounded;
    const bool changed = !terminal && pl.has_change;
    if (changed) {
      // A deferred plan still open here (Startup's batch plan when the batch
      // changed nothing) describes the model this rule replaces: retire it,
      // so the next deferred rule starts a fresh plan on the new model.
      if (active) {
        if (pending) throw std::logic_error("materialized rule over a plan with unapplied changes");
        active = reshaped = false;
        plan = Plan{};
        stats = Stats{};
      }
      apply(pl, false);
      out.trace.push_back(std::string("apply=") + name);
    }
    if (pl.has_new_A) free_csr(pl.new_A);
    return changed;
  }
};

bool good_progress(int64_t before, int64_t after, int64_t d) { return before >= d && after <= before - d; }

}  // namespace

void run_presolve(const gpp_lp& input, const gpp_params& p, PresolveOutput& out, SchedulePolicy* policy,
                  std::vector<RoundRecord>* trace) {
  const NvtxRange range("presolve");
  Engine e(p, out);
  WorkingLp& cur = e.cur;
  cur.A = DevCsr{input.A.rows, input.A.cols, input.A.nnz, input.A.rowPtr, input.A.colVal, input.A.nzVal};
  cur.AT = DevCsr{input.AT.rows, input.AT.cols, input.AT.nnz, input.AT.rowPtr, input.AT.colVal, input.AT.nzVal};
  cur.c = input.c; cur.AL = input.AL; cur.AU = input.AU; cur.l = input.l; cur.u = input.u;
  cur.obj = input.obj_constant;
  cur.owns = false;
  out.original_rows = cur.m();
  out.original_cols = cur.n();
  init_record(out.record, cur.m(), cur.n());
  invalidate_schedules();
  ctx().sync("presolve initialization");
  const auto t0 = std::chrono::steady_clock::now();
  const bool has_time_limit = p.max_time > 0.0 && std::isfinite(p.max_time);
  auto time_exceeded = [&]() {
    return has_time_limit &&
           std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count() >= p.max_time;
  };

  if (p.enable_startup && p.max_iters > 0 && !time_exceeded()) {
    // Startup (gpu_presolve.cu:2361-2454): the structure-specific rules, all
    // off when enable_structure_specific_rules is (:2088-2094).  Column
    // domination, two-row variable elimination and zero-cost product
    // variables share one plan, each seeing the deletions of those before it,
    // and the plan is applied once; then the variable-pair reformulation
    // (:2416-2445) and the absolute-value reformulation, gated by its prefix
    // screen (:2447), each on its own materialised plan.  The phase consumes
    // one iteration (:2453).
    const bool batch = p.enable_structure_specific_rules &&
                       (p.enable_column_domination || p.enable_two_row_variable_elimination ||
                        p.enable_zero_cost_product_variables);
    if (batch && e.deferred_rule(true, "startup_projection_batch", [&] {
          if (p.enable_column_domination) rule_column_domination(e.plan, cur, p);
          if (p.enable_two_row_variable_elimination && !time_exceeded())
            rule_two_row_variable_elimination(e.plan, cur, p);
          if (p.enable_zero_cost_product_variables && !time_exceeded())
            rule_zero_cost_product_variables(e.plan, cur, p);
        }))
      e.materialize("startup");
    if (p.enable_structure_specific_rules && p.enable_piecewise_linear_reformulation_variable_pair && !e.terminal &&
        !time_exceeded())
      e.materialized_rule(true, "startup_piecewise_linear_reformulation_variable_pair",
                          [&](Plan& pl) { rule_variable_pair(pl, cur, p); });
    if (p.enable_structure_specific_rules && p.enable_piecewise_linear_reformulation_absolute_value &&
        !e.terminal && !time_exceeded() && absolute_value_prefix_screen(cur))
      e.materialized_rule(true, "startup_piecewise_linear_reformulation_absolute_value",
                          [&](Plan& pl) { rule_absolute_value(pl, cur, p); });
    ++out.iterations;
  }
  auto deferred = [&](bool enabled, const char* name, auto rule) {
    return !time_exceeded() && e.deferred_rule(enabled, name, rule);
  };
  // Round schedule: `skip` gates rules for the current round (a policy's
  // choice; 0 in the plain loop), `ran` / `changed` record what the gated
  // rules did.
  uint32_t skip = 0, ran = 0, changed_rules = 0;
  auto gate = [&](int rule, bool enabled) {
    const bool run = enabled && !(skip >> rule & 1u);
    if (run) ran |= 1u << rule;
    return run;
  };
  auto note = [&](int rule, bool ch) {
    if (ch) changed_rules |= 1u << rule;
    return ch;
  };
  auto cleanup = [&]() {
    out.trace.push_back("phase=cleanup");
    // The first four rules' first checks run at once on the plan as it stands
    // (one readback instead of four).  While every rule so far has changed
    // nothing the plan is still the probed one, so a rule whose check found
    // nothing is passed over; from the first rule that changes the plan on,
    // the rules run as usual.
    uint32_t may = ~0u;
    const uint32_t probed = (p.enable_infeasible_and_fixed_variables ? kProbeFixed : 0u) |
                            (p.enable_empty_columns ? kProbeEmptyColumns : 0u) |
                            (p.enable_empty_rows ? kProbeEmptyRows : 0u) |
                            (p.enable_singleton_rows ? kProbeSingletonRows : 0u);
    // Singleton columns' test goes along with the probe (not under a time
    // limit, which may end the round between the two).
    const bool columns = gate(kGateSingletonColumns, p.enable_singleton_columns);
    SingletonTest ahead;
    if (probed && !e.terminal && !time_exceeded()) {
      e.prepare();
      e.refresh();
      may = cleanup_probe(e.plan, cur, e.stats, p, probed, columns && !has_time_limit ? &ahead : nullptr);
      if (may) ahead.asked = false;   // its kernels did nothing
    }
    bool quiet = true;
    auto step = [&](uint32_t bit, bool enabled, const char* name, auto rule) {
      if (quiet && !(may & bit)) return !time_exceeded() && e.skipped_rule(enabled, name);
      const bool changed = deferred(enabled, name, rule);
      quiet = quiet && !changed;
      return changed;
    };
    bool ch = step(kProbeFixed, p.enable_infeasible_and_fixed_variables, "infeasible_and_fixed_variables",
                   [&] { rule_fixed_variables(e.plan, cur, p); });
    ch = step(kProbeEmptyColumns, p.enable_empty_columns, "empty_columns",
              [&] { rule_empty_columns(e.plan, cur, e.stats, p); }) || ch;
    ch = step(kProbeEmptyRows, p.enable_empty_rows, "empty_rows", [&] { rule_empty_rows(e.plan, cur, e.stats, p); }) ||
         ch;
    ch = step(kProbeSingletonRows, p.enable_singleton_rows, "singleton_rows",
              [&] { rule_singleton_rows(e.plan, cur, e.stats, p); }) || ch;
    ch = note(kGateSingletonColumns,
              deferred(columns, "singleton_columns",
                       [&] { rule_singleton_columns(e.plan, cur, e.stats, p, &ahead); })) || ch;
    return ch;
  };
  auto propagation = [&]() {
    out.trace.push_back("phase=propagation");
    bool bounds_changed = false;
    if (gate(kGateBoundStrengthening, p.enable_bound_strengthening) && !e.terminal && !time_exceeded()) {
      e.prepare();
      bounds_changed = note(kGateBoundStrengthening,
                            e.deferred_rule(true, "bound_strengthening",
                                            [&] { rule_bound_strengthening(e.plan, cur, e.stats, p); }));
    }
    const bool tail = gate(kGateRedundantRowsDualFix, p.enable_infeasible_and_redundant_rows || p.enable_dual_fix);
    e.plan.row_kinds_current = false;
    DualFixTest ahead;
    bool tail_changed =
        deferred(tail && p.enable_infeasible_and_redundant_rows, "infeasible_and_redundant_rows",
                 [&] { rule_redundant_rows(e.plan, cur, e.stats, p, p.enable_dual_fix ? &ahead : nullptr); });
    tail_changed = deferred(tail && p.enable_dual_fix, "dual_fix",
                            [&] { rule_dual_fix(e.plan, cur, e.stats, p, &ahead); }) ||
                   tail_changed;
    note(kGateRedundantRowsDualFix, tail_changed);
    return bounds_changed;
  };

  enum Phase { Cleanup, Propagation, Aggregation, Parallel } phase = Cleanup;
  const int64_t min_dec = 100;
  int bound_only_rounds = 0;
  const int64_t initial_live = p.max_iters > 0 && !e.terminal && !time_exceeded() ? e.live_nnz() : 0;
  const int configured = std::max(1, p.bound_strengthening_max_bound_only_rounds);
  int limit = configured;
  if (p.bound_strengthening_bound_only_nnz_round_budget > 0 && initial_live > 0)
    limit = int(std::min<int64_t>(limit, std::max<int64_t>(1, p.bound_strengthening_bound_only_nnz_round_budget / initial_live)));
  {
    const int64_t m = cur.m(), n = cur.n();
    if (m >= 512 && m <= 2048 && n >= 128 * m && n <= 256 * m && initial_live >= 2048 * m && initial_live <= 8192 * m)
      limit = std::max(limit, std::min(2, configured));
  }
  // Host-side state of the round features.
  const int64_t initial_rows = std::max<int64_t>(1, cur.m());
  const int64_t initial_nnz_all = std::max<int64_t>(1, initial_live);
  int64_t removed_prev = 0, removed_prev2 = 0;
  int round = 0;
  bool last_changed[kGatedRules] = {};
  int last_ran[kGatedRules];
  for (int& r : last_ran) r = -1;
  const bool scheduled = policy || trace;
  DBuf<uint32_t> inf_hist;
  if (scheduled) {
    inf_hist.alloc(8, ctx().stream);
    inf_hist.zero();
    e.inf_hist = inf_hist.p;
    if (e.active) e.plan.inf_hist = inf_hist.p;
  }
  while (p.max_iters > 0 && !e.terminal && !time_exceeded()) {
    if (phase != Cleanup) {
      if (out.iterations >= p.max_iters) { out.stopped_at_iteration_limit = true; break; }
      ++out.iterations;
    }
    // Cleanup does not use the nnz before it (outside traced runs); the other
    // phases read it after their own waits.
    Engine::LaterCount before_count;
    if (scheduled) before_count.known = e.live_nnz();
    else if (phase != Cleanup) before_count = e.live_nnz_later();
    const auto before_nnz = [&]() { return e.value(before_count); };
    RoundRecord rec;
    skip = ran = changed_rules = 0;
    if (scheduled) {
      float* f = rec.features;
      f[int(phase)] = 1.0f;
      f[4] = float(round) / 32.0f;
      f[5] = float(double(before_count.known) / double(initial_nnz_all));
      f[6] = float(double(removed_prev) / double(initial_nnz_all));
      f[7] = float(double(removed_prev2) / double(initial_nnz_all));
      for (int g = 0; g < kGatedRules; ++g) {
        f[8 + g] = last_changed[g] ? 1.0f : 0.0f;
        f[14 + g] = last_ran[g] < 0 ? 1.0f : std::min(1.0f, float(round - last_ran[g]) / 16.0f);
      }
      f[20] = float(bound_only_rounds) / 8.0f;
      f[21] = float(std::log10(double(initial_nnz_all)) / 8.0);
      f[22] = float(1.0 - double(before_count.known) / double(initial_nnz_all));
      f[23] = float(double(cur.m()) / double(initial_rows));
      const std::vector<uint32_t> h = to_host(inf_hist.p, 8);
      for (int side = 0; side < 2; ++side) {
        const double rows = double(h[4 * side] + h[4 * side + 1] + h[4 * side + 2] + h[4 * side + 3]);
        for (int k = 0; k < 4; ++k) f[24 + 4 * side + k] = rows > 0 ? float(double(h[4 * side + k]) / rows) : 0.0f;
      }
      rec.phase = int32_t(phase);
      rec.iteration = out.iterations;
      rec.nnz_before = before_count.known;
      if (policy) {
        bool stop = false;
        skip = policy->decide(f, &stop);
        if (stop) break;
      }
    }
    if (phase == Cleanup) {
      const uint64_t ser = e.deletion_serial;
      const bool changed = cleanup();
      if (e.deletion_serial != ser) bound_only_rounds = 0;
      phase = changed ? Cleanup : Propagation;
    } else if (phase == Propagation) {
      const uint64_t ser = e.deletion_serial;
      const bool bounds_changed = propagation();
      bound_only_rounds = e.deletion_serial != ser ? 0 : bound_only_rounds + 1;
      e.materialize("1");
      const int64_t after = e.live_nnz();
      const bool nnz_progress = good_progress(before_nnz(), after, min_dec);
      const bool bound_progress = bounds_changed && bound_only_rounds < limit;
      phase = nnz_progress || bound_progress ? Cleanup : Aggregation;
      if (phase == Aggregation) bound_only_rounds = 0;
    } else if (phase == Aggregation) {
      out.trace.push_back("phase=aggregation");
      if (!time_exceeded() && gate(kGateDoubleton, p.enable_doubleton_equations))
        e.materialized_rule(true, "doubleton_equations", [&](Plan& pl) { rule_doubleton_equations(pl, cur, p); });
      const int64_t after = e.live_nnz();
      const int64_t before = before_nnz();
      note(kGateDoubleton, after < before);
      phase = good_progress(before, after, min_dec) ? Cleanup : Parallel;
    } else {
      out.trace.push_back("phase=parallel");
      bool changed = note(kGateParallelRows,
                          deferred(gate(kGateParallelRows, p.enable_parallel_rows), "parallel_rows",
                                   [&] { rule_parallel_rows(e.plan, cur, e.stats, p); }));
      changed = note(kGateParallelColumns,
                     deferred(gate(kGateParallelColumns, p.enable_parallel_columns), "parallel_columns",
                              [&] { rule_parallel_columns(e.plan, cur, e.stats, p); })) || changed;
      e.materialize("2");
      const int64_t after = e.live_nnz();
      const int64_t before = before_nnz();
      const bool stop_loop = !(changed && good_progress(before, after, min_dec));
      if (scheduled) {
        rec.ran = ran; rec.changed = changed_rules; rec.nnz_after = after;
        if (trace) trace->push_back(rec);
      }
      if (stop_loop) break;
      phase = Cleanup;
      if (scheduled) {
        removed_prev2 = removed_prev;
        removed_prev = before - after;
        for (int g = 0; g < kGatedRules; ++g)
          if (ran >> g & 1u) { last_ran[g] = round; last_changed[g] = (changed_rules >> g & 1u) != 0; }
        ++round;
      }
      continue;
    }
    if (scheduled) {
      const int64_t after = e.live_nnz();
      rec.ran = ran; rec.changed = changed_rules; rec.nnz_after = after;
      if (trace) trace->push_back(rec);
      removed_prev2 = removed_prev;
      removed_prev = before_count.known - after;
      for (int g = 0; g < kGatedRules; ++g)
        if (ran >> g & 1u) { last_ran[g] = round; last_changed[g] = (changed_rules >> g & 1u) != 0; }
      ++round;
    }
  }
  e.materialize("finalize");
  e.save_vectors();
  settle_fixed(out.record);
  globalize_segments(out.record);
  ctx().sync("presolve finalize");
  out.reduced_rows = cur.m();
  out.reduced_cols = cur.n();
  out.reduced_nnz = cur.A.nnz;
  out.obj_constant_delta = cur.obj - input.obj_constant;
  out.elapsed_seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  out.has_change = cur.owns;
  out.reduced = cur;      // ownership moves to the output when cur.owns
  out.owns_reduced = cur.owns;
  cur.owns = false;
}

}  // namespace gpp

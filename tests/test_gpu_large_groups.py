"""Hash groups and rows past the sizes that one thread or warp takes, against
the oracle bit for bit: groups of equal columns around 8 (one thread) and 32
(a warp's partners at once) whose bounds and costs make pairs merge, fix one
side, or do nothing; rows around 1,024 entries for the row hash; more
acceptable doubleton rows than one block matches."""
import numpy as np
import pytest

import pyoracle
from gpp_b200 import capi, device, lpgen
from test_gpu_pipeline import assert_same

pytestmark = pytest.mark.gpu


def group_lp(size, seed):
    """Columns 0 .. size-1 are multiples of one two-entry pattern; the rest tie
    the rows down.  Costs follow the multiple for two in three columns (those
    merge); a few upper bounds are infinite, and with an odd seed some lower ones
    too (most of those models are unbounded)."""
    rng = np.random.default_rng(seed)
    extra = 6
    n, m = size + extra, 4
    ratio = np.where(rng.random(size) < 0.3, -1.0, 1.0) * rng.choice([0.5, 1.0, 1.0, 2.0], size=size)
    ratio[0] = 1.0
    rows = np.concatenate([np.zeros(size), np.ones(size), np.repeat(np.arange(4), extra)]).astype(np.int64)
    cols = np.concatenate([np.arange(size), np.arange(size), np.tile(np.arange(size, n), 4)]).astype(np.int64)
    vals = np.concatenate([ratio, -3.0 * ratio, rng.uniform(0.5, 2.0, size=4 * extra)])
    p, i, v = lpgen.coo_to_csr(m, rows, cols, vals)
    c = np.where(rng.random(size) < 0.67, ratio, ratio + rng.uniform(0.1, 2.0, size=size))
    lo, hi = np.zeros(size), rng.uniform(1.0, 4.0, size=size)
    hi[(rng.random(size) < 4.0 / size) & (ratio > 0)] = np.inf
    if seed % 2:
        lo[rng.random(size) < 2.0 / size] = -np.inf
    c = np.concatenate([c, rng.uniform(0.5, 1.0, size=extra)])
    lo = np.concatenate([lo, np.zeros(extra)])
    hi = np.concatenate([hi, np.full(extra, 9.0)])
    return lpgen.HostLP(m, n, p, i, v, c, np.full(m, -50.0), np.full(m, 50.0), lo, hi).ensure_transpose()


def compare(lp, params):
    dlp = device.DeviceLp(lp)
    s = device.preprocess(dlp, params)
    try:
        orc = pyoracle.presolve(lp, params)
        if s.has_unbounded or s.has_infeasible:
            assert (s.has_unbounded, s.has_infeasible) == (orc.summary.has_unbounded, orc.summary.has_infeasible)
        else:
            assert_same(device.Result(s), orc)
    finally:
        device.free_summary(s)


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("size", [2, 7, 8, 9, 10, 31, 33, 34, 65, 300])
def test_column_groups(size, seed):
    params = capi.params_with_rules(["parallel_columns"], enable_folding=0, enable_startup=0,
                                    parallel_columns_scale_guard_min_groups=0)
    compare(group_lp(size, 100 * size + seed), params)


@pytest.mark.parametrize("hubs", [1, 12])
def test_long_rows_hash(hubs):
    lp = lpgen.random_lp(3000, 7000, seed=hubs, hub_rows=hubs)
    compare(lp, capi.params_with_rules(["singleton_rows", "parallel_rows"], enable_folding=0, enable_startup=0))


def repeated_rows_lp(copies, longest, seed):
    """Every row comes `copies` times, scaled, among rows of 9 to `longest`
    entries in no order; some columns are fixed (dead under the hash's mask),
    first and last ones of rows among them."""
    rng = np.random.default_rng(seed)
    n = 3 * longest
    rows, cols, vals, at = [], [], [], 0
    for length in rng.permutation(np.arange(9, longest + 1)):
        col = np.sort(rng.choice(n, size=length, replace=False))
        val = rng.choice([1.0, -2.0, 0.5], size=length)
        for k in range(copies):
            rows.append(np.full(length, at))
            cols.append(col)
            vals.append(val * (1.0, 2.0, -0.5)[k % 3])
            at += 1
    order = rng.permutation(at)
    p, i, v = lpgen.coo_to_csr(at, order[np.concatenate(rows)], np.concatenate(cols), np.concatenate(vals))
    hi = np.where(rng.random(n) < 0.15, 0.0, 5.0)
    return lpgen.HostLP(at, n, p, i, v, rng.uniform(0.5, 1.0, size=n), np.full(at, -900.0), np.full(at, 900.0),
                        np.zeros(n), hi).ensure_transpose()


@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("copies,longest", [(1, 16), (2, 17), (3, 33), (2, 70), (3, 1030)])
def test_row_hash_of_mixed_lengths(copies, longest, fixed):
    rules = ["parallel_rows"] + (["infeasible_and_fixed_variables"] if fixed else [])
    compare(repeated_rows_lp(copies, longest, longest), capi.params_with_rules(rules, enable_folding=0, enable_startup=0))


@pytest.mark.parametrize("m", [3000, 120000])
def test_doubleton_matching(m):
    compare(lpgen.random_lp(m, int(2.5 * m), seed=1),
            capi.params_with_rules(["doubleton_equations"], enable_folding=0, enable_startup=0,
                                   doubleton_equations_min_selected_per_batch=1,
                                   doubleton_equations_min_selected_ratio=0.0))

"""Bound finalisation where it needs the largest |a| of a column: columns around the
lengths that a thread (64 stored entries), a warp (1,024) and a block take, whose
candidates nearly meet, so that one entry decides whether they are fixed; the entry
stands first, last or in a removed row; against the oracle bit for bit."""
import numpy as np
import pytest

from gpp_b200 import capi, lpgen
from test_gpu_dense_models import kernels_of, presolve
from test_gpu_large_groups import compare

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 6, 7, 63, 64, 65, 66, 127, 1023, 1024, 1025, 1026, 1100, 2048, 2049, 5000]


def nearly_closed(place, gap, seed):
    """Per length a column x with a companion t in [0, gap], under x + t <= 5 and x + t >= 5,
    and `length` - 2 further entries of at most 1 in loose rows, but for one of 100."""
    rng = np.random.default_rng(seed)
    k, wide = len(LENGTHS), max(LENGTHS)
    rows, cols, vals = [], [], []
    for j, length in enumerate(LENGTHS):
        size = max(length - 2, 0)
        r = np.sort(rng.choice(wide, size, replace=False))
        v = rng.uniform(0.5, 1.0, size)
        if size:
            v[{"first": 0, "last": -1, "middle": size // 2}[place]] = 100.0
        rows.append(r); cols.append(np.full(size, j)); vals.append(v)
    pair = wide + np.arange(2 * k)
    rows += [pair, pair]
    cols += [np.tile(np.arange(k), 2), k + np.tile(np.arange(k), 2)]
    vals += [np.ones(2 * k), np.ones(2 * k)]
    m = wide + 2 * k
    p, i, v = lpgen.coo_to_csr(m, *(np.concatenate(a) for a in (rows, cols, vals)))
    AL, AU = np.full(m, -np.inf), np.full(m, 1e7)
    AU[wide:wide + k], AU[wide + k:], AL[wide + k:] = 5.0, np.inf, 5.0
    u = np.concatenate([np.full(k, 10.0), np.full(k, gap)])
    return lpgen.HostLP(m, 2 * k, p, i, v, rng.standard_normal(2 * k), AL, AU, np.zeros(2 * k), u).ensure_transpose()


@pytest.mark.parametrize("place", ["first", "last", "middle"])
@pytest.mark.parametrize("gap", [1e-12, 1e-7, 1e-4])   # all fixed, those without the large entry, none
def test_one_entry_decides(place, gap):
    lp = nearly_closed(place, gap, seed=len(place))
    only = capi.params_with_rules(["bound_strengthening"], enable_folding=0, enable_startup=0)
    compare(lp, only)
    compare(lp, capi.params_with_rules(["bound_strengthening"], enable_folding=0, enable_startup=0, record_postsolve_tape=0))
    compare(lp, capi.Params.defaults(enable_folding=0))
    deferred = any("finalize_deferred" in k for k in kernels_of(presolve(lp, only)))
    assert deferred == (gap < 1e-6 and not (gap == 1e-7 and place == "first"))


def test_columns_whose_bounds_cross():
    lp = nearly_closed("last", 1e-7, seed=1)
    lp.AU[lp.m - 2 * len(LENGTHS):lp.m - len(LENGTHS)] = 4.0   # x + t <= 4 and >= 5
    compare(lp, capi.params_with_rules(["bound_strengthening"], enable_folding=0, enable_startup=0))

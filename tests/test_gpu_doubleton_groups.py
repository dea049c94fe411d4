"""Doubleton equations whose columns and rows lie on both sides of what eight lanes
take (64 entries): shifted, substituted and rebuilt rows of 9 to a few thousand
entries, eliminated and kept columns in up to 300 rows; against the oracle bit for
bit."""
import numpy as np
import pytest

from gpp_b200 import capi, lpgen
from test_gpu_large_groups import compare

pytestmark = pytest.mark.gpu


def lp_with_wide_columns(entries, hubs, seed):
    """A random LP to which equations x_j + a x_k = b are added for columns that also
    appear in `entries` further rows (j, k or both), some of them fixed by theirs."""
    rng = np.random.default_rng(seed)
    base = lpgen.random_lp(600, 1500, seed=seed, hub_rows=hubs)
    m, n = base.m, base.n
    rows = [np.repeat(np.arange(m), np.diff(base.row_ptr))]
    cols, vals = [base.col_idx.astype(np.int64)], [base.values]
    AL, AU = list(base.AL), list(base.AU)
    pairs = 24
    for q in range(pairs):
        j, k = n + 2 * q, n + 2 * q + 1
        rows.append(np.full(2, len(AL)))
        cols.append(np.array([j, k]))
        vals.append(np.array([1.0, -1.0 if q % 3 else 2.0]))
        b = float(rng.integers(0, 3))
        AL.append(b)
        AU.append(b)
        wide = entries if q % 4 == 0 else 5
        for side in ([j], [k], [j, k])[q % 3]:
            touched = rng.choice(m, size=min(wide, m), replace=False)
            rows.append(np.sort(touched))
            cols.append(np.full(touched.size, side))
            vals.append(rng.choice([1.0, 0.5, -2.0], size=touched.size))
    total = n + 2 * pairs
    p, i, v = lpgen.coo_to_csr(len(AL), np.concatenate(rows), np.concatenate(cols), np.concatenate(vals))
    lo = np.concatenate([base.l, np.zeros(2 * pairs)])
    hi = np.concatenate([base.u, rng.choice([3.0, 6.0], size=2 * pairs)])
    c = np.concatenate([base.c, rng.uniform(-1.0, 1.0, size=2 * pairs)])
    return lpgen.HostLP(len(AL), total, p, i, v, c, np.array(AL), np.array(AU), lo, hi).ensure_transpose()


@pytest.mark.parametrize("hubs", [0, 8])
@pytest.mark.parametrize("entries", [9, 63, 64, 65, 300])
def test_doubleton_groups(entries, hubs):
    compare(lp_with_wide_columns(entries, hubs, entries),
            capi.params_with_rules(["doubleton_equations"], enable_folding=0, enable_startup=0,
                                   doubleton_equations_min_selected_per_batch=1,
                                   doubleton_equations_min_selected_ratio=0.0,
                                   doubleton_equations_max_fill_in_proxy=1000000))

"""Doubleton equations by the number of columns and rows that share a warp: one, two or
four of them, with counts around the lines (2,368 and 4,736) and long ones that take a
warp each past those; against the oracle bit for bit."""
import numpy as np
import pytest

from gpp_b200 import capi, lpgen
from test_gpu_large_groups import compare

pytestmark = pytest.mark.gpu


def paired_lp(m, n, per, pairs, wide, seed):
    """m rows of `per` of n columns, and `pairs` equations x - a y = b of further columns,
    which also stand in `wide` of the rows."""
    rng = np.random.default_rng(seed)
    first = rng.integers(0, n, m)
    step = n // per
    rows = [np.repeat(np.arange(m), per), np.repeat(m + np.arange(pairs), 2)]
    cols = [((first[:, None] + np.arange(per) * step) % n).ravel(), n + np.arange(2 * pairs)]
    vals = [rng.uniform(0.5, 2.0, m * per), np.column_stack([np.ones(pairs), rng.choice([-1.0, 2.0], pairs)]).ravel()]
    touched = (rng.integers(0, m, 2 * pairs)[:, None] + np.arange(wide) * (m // wide)) % m
    rows.append(touched.ravel())
    cols.append(np.repeat(n + np.arange(2 * pairs), wide))
    vals.append(rng.choice([1.0, 0.5, -2.0], touched.size))
    total, b = n + 2 * pairs, rng.integers(0, 3, pairs).astype(float)
    p, i, v = lpgen.coo_to_csr(m + pairs, *(np.concatenate(a) for a in (rows, cols, vals)))
    wide_side = np.full(m, 40.0 * per)
    return lpgen.HostLP(m + pairs, total, p, i, v, rng.uniform(-1.0, 1.0, total), np.concatenate([-wide_side, b]),
                        np.concatenate([wide_side, b]), np.zeros(total), np.full(total, 6.0)).ensure_transpose()


@pytest.mark.parametrize("m,n,per,pairs,wide", [
    (3000, 4000, 6, 2368, 3), (2400, 4000, 6, 2369, 3),       # one and two columns to a warp
    (3000, 4000, 6, 4736, 4), (3000, 4000, 6, 4737, 4),       # two and four
    (2500, 6000, 72, 60, 90), (200, 9000, 3000, 20, 150),     # long rows and columns, a warp each
])
def test_doubleton_counts(m, n, per, pairs, wide):
    compare(paired_lp(m, n, per, pairs, wide, pairs),
            capi.params_with_rules(["doubleton_equations"], enable_folding=0, enable_startup=0,
                                   doubleton_equations_min_selected_per_batch=1,
                                   doubleton_equations_min_selected_ratio=0.0,
                                   doubleton_equations_max_fill_in_proxy=1000000))

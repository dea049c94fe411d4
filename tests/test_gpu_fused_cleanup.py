"""The Cleanup probe with singleton columns behind it, as one cluster (up to 8,192
rows and columns) and as a chain of launches, on both sides of that line and at the
smallest models: columns that are substituted out, rows of more than 1,024
entries that hold a candidate, an unbounded candidate, a time limit (under which the
two are asked one after the other); against the oracle bit for bit."""
import numpy as np
import pytest

from gpp_b200 import capi, lpgen
from test_gpu_large_groups import compare

pytestmark = pytest.mark.gpu

RULES = ["infeasible_and_fixed_variables", "empty_rows", "empty_columns", "singleton_rows", "singleton_columns"]


def params(**extra):
    return capi.params_with_rules(RULES, enable_folding=0, enable_startup=0, **extra)


@pytest.mark.parametrize("n", [1, 2, 33, 2048, 2049, 8191, 8192, 8193, 16400])
def test_slack_columns(n):
    lp = lpgen.random_lp(max(1, n // 3), max(1, n - n // 3), seed=n, slack_frac=0.9) if n > 2 else None
    if lp is None:
        p, i, v = lpgen.coo_to_csr(1, np.zeros(n, np.int64), np.arange(n), np.ones(n))
        lp = lpgen.HostLP(1, n, p, i, v, np.arange(1.0, n + 1), np.zeros(1), np.ones(1), np.zeros(n),
                          np.full(n, np.inf)).ensure_transpose()
    compare(lp, params())
    compare(lp, params(max_time=1000.0))
    compare(lp, capi.Params.defaults(enable_folding=0))


@pytest.mark.parametrize("m,n,hubs", [(2000, 6000, 5), (3000, 9000, 40)])
def test_candidates_in_long_rows(m, n, hubs):
    compare(lpgen.random_lp(m, n, seed=hubs, hub_rows=hubs, slack_frac=0.5), params())


@pytest.mark.parametrize("n", [40, 9000])
def test_unbounded_candidate(n):
    lp = lpgen.random_lp(n // 2, n, seed=3, slack_frac=0.3)
    lp.ensure_transpose()
    j = int(np.flatnonzero(np.diff(lp.at_ptr) == 1)[-1])
    row = lp.at_idx[lp.at_ptr[j]]
    lp.values[np.arange(lp.row_ptr[row], lp.row_ptr[row + 1])[lp.col_idx[lp.row_ptr[row]:lp.row_ptr[row + 1]] == j]] = 1.0
    lp.AL[row], lp.l[j], lp.u[j], lp.c[j] = -np.inf, -np.inf, np.inf, 1.0
    lp.at_ptr = None
    compare(lp.ensure_transpose(), params())

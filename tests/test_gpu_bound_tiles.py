"""Bound strengthening at the edges of its tiles of 256 columns (and of the 1,024
tiles whose record counts are summed at once): few, some, all columns move,
with and without a supporting row, against the oracle bit for bit."""
import numpy as np
import pytest

from gpp_b200 import capi, lpgen
from test_gpu_large_groups import compare

pytestmark = pytest.mark.gpu


def pair_lp(n, share, seed):
    """Row i holds columns i and i + 1; a share of the rows is tight enough to
    imply bounds on both, some columns start out free above, some fixed."""
    rng = np.random.default_rng(seed)
    m = n - 1
    rows = np.repeat(np.arange(m), 2)
    cols = (rows + np.tile([0, 1], m)).astype(np.int64)
    vals = rng.choice([1.0, 2.0, -1.0], size=2 * m)
    p, i, v = lpgen.coo_to_csr(m, rows, cols, vals)
    tight = rng.random(m) < share
    hi = np.where(rng.random(n) < 0.2, np.inf, rng.integers(3, 9, size=n).astype(float))
    return lpgen.HostLP(m, n, p, i, v, rng.uniform(-1.0, 1.0, size=n), np.full(m, -100.0),
                        np.where(tight, rng.integers(1, 6, size=m), 100).astype(float), np.zeros(n),
                        hi).ensure_transpose()


@pytest.mark.parametrize("share", [0.0, 0.02, 1.0])
@pytest.mark.parametrize("n", [2, 255, 256, 257, 511, 513, 256 * 1024 - 1, 256 * 1024 + 1])
def test_bounds_at_tile_edges(n, share):
    for tape in (1, 0):
        compare(pair_lp(n, share, n), capi.params_with_rules(["bound_strengthening"], enable_folding=0,
                                                             enable_startup=0, record_postsolve_tape=tape))


@pytest.mark.parametrize("entries", [63, 64, 65, 128, 129, 1500])
def test_bounds_of_wide_columns(entries):
    """Three columns of `entries` entries each whose bounds every row implies anew
    (their largest coefficient decides whether they get fixed), some rows redundant."""
    rng = np.random.default_rng(entries)
    m, n = entries, entries + 3
    rows = np.repeat(np.arange(m), 4)
    cols = np.stack([np.zeros(m), np.ones(m), np.full(m, 2.0), 3 + np.arange(m)], axis=1).astype(np.int64).ravel()
    vals = rng.choice([1.0, 2.0, 0.5], size=4 * m)
    p, i, v = lpgen.coo_to_csr(m, rows, cols, vals)
    lp = lpgen.HostLP(m, n, p, i, v, rng.uniform(-1.0, 1.0, size=n), np.full(m, -np.inf),
                      np.where(rng.random(m) < 0.5, rng.integers(2, 9, size=m), 500).astype(float), np.zeros(n),
                      rng.choice([4.0, np.inf], size=n)).ensure_transpose()
    compare(lp, capi.params_with_rules(["bound_strengthening", "infeasible_and_redundant_rows"], enable_folding=0,
                                       enable_startup=0))

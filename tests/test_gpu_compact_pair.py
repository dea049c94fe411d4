"""The compaction of A and A^T in one launch, as a presolve does it, at the edges of its
tiles: entry counts around 256 (a warp's part) and 2,048 (a tile), rows or columns that
start and end there, runs of empty ones before, at and past the last entry, and rows long
enough (33 parts) that their warp marks the parts; against the oracle bit for bit."""
import numpy as np
import pytest

from gpp_b200 import capi, lpgen
from test_gpu_large_groups import compare
from test_gpu_tile_edges import model

pytestmark = pytest.mark.gpu


def lp_of(layout, nnz, transposed, seed):
    """Columns with equal bounds and free rows go; nothing else does."""
    rng = np.random.default_rng(seed)
    m, n, row_ptr, idx, values = model(layout, nnz, rng)
    rows = np.repeat(np.arange(m), np.diff(row_ptr))
    if transposed:
        m, n, rows, idx = n, m, idx, rows
    p, i, v = lpgen.coo_to_csr(m, rows, idx, values)
    side = np.where(rng.random(m) < 0.4, np.inf, 0.25)
    bound = np.where(rng.random(n) < 0.3, 0.0, 1.0)
    return lpgen.HostLP(m, n, p, i, v, rng.standard_normal(n), np.where(np.isinf(side), -side, side), side, -bound,
                        bound).ensure_transpose()


@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("layout", ["one row", "rows of 32", "edges", "random"])
@pytest.mark.parametrize("nnz", [255, 256, 257, 2047, 2048, 2049, 32 * 256, 33 * 256, 33 * 256 + 1, 34 * 256 + 1, 40_000])
def test_both_matrices_at_tile_edges(nnz, layout, transposed):
    lp = lp_of(layout, nnz, transposed, nnz)
    compare(lp, capi.params_with_rules(["infeasible_and_fixed_variables", "infeasible_and_redundant_rows"],
                                       enable_folding=0, enable_startup=0))

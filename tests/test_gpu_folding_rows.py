"""Folding of dense symmetric models against the oracle, colours and folded model bit for
bit: rows around the lengths that a lane (16 entries), a warp (1,024) and a block take, in
models of one row to a warp (up to 9,472 rows or columns), two and four."""
import numpy as np
import pytest

from gpp_b200 import lpgen
from rule_cases import Run, bits

pytestmark = pytest.mark.gpu


def copied_block(lengths, width, copies, seed):
    """`copies` equal blocks: rows of the given lengths over `width` columns."""
    rng = np.random.default_rng(seed)
    idx = np.concatenate([np.sort(rng.choice(width, k, replace=False)) for k in lengths])
    rows, m0 = np.repeat(np.arange(len(lengths)), lengths), len(lengths)
    val = np.round(rng.uniform(1.0, 10.0, idx.size), 3)
    shift = np.repeat(np.arange(copies), idx.size)
    p, i, v = lpgen.coo_to_csr(m0 * copies, np.tile(rows, copies) + m0 * shift, np.tile(idx, copies) + width * shift,
                               np.tile(val, copies))
    side = np.tile(np.bincount(rows, weights=val, minlength=m0) * 1.5, copies)
    return lpgen.HostLP(m0 * copies, width * copies, p, i, v, np.tile(rng.standard_normal(width), copies),
                        np.full(side.size, -np.inf), side, np.zeros(width * copies),
                        np.tile(rng.uniform(1.0, 9.0, width), copies)).ensure_transpose()


@pytest.mark.parametrize("lengths,width,copies", [
    ([15, 16, 17, 31, 32, 33, 64, 65], 70, 5), ([1, 1023, 1024, 1025, 1026], 1100, 3), ([40] * 30, 60, 200),
    ([20] * 30, 50, 190), ([18] * 33, 40, 600)])
def test_dense_blocks_fold_as_the_oracle(lengths, width, copies):
    lp = copied_block(lengths, width, copies, seed=len(lengths))
    g = Run("gpu", lp, [], enable_folding=1, max_iters=0)
    o = Run("oracle", lp, [], enable_folding=1, max_iters=0)
    assert g.s.folding_applied == 1 and o.s.folding_applied == 1
    for a, b in zip(g.fold, o.fold):
        assert np.array_equal(a, b)
    for k in ("A_ptr", "A_idx", "A_val", "c", "l", "u", "AL", "AU"):
        a, b = getattr(g, k), getattr(o, k)
        assert np.array_equal(bits(a), bits(b)) if a.dtype == np.float64 else np.array_equal(a, b), k

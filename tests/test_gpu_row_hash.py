"""Row hashes of both modes against the oracle's: rows around the lengths at which a
thread, a group of lanes and a block take over (8, 32, 1,024 stored entries and the
rounds of each), under column masks, with removed rows, pivots at the tolerance,
infinities and NaN."""
import ctypes as C

import numpy as np
import pytest

import pyoracle
from gpp_b200 import capi, lpgen
from gpp_b200.device import _raise, ptr, to_device
from test_gpu_dense_models import dense_lp, kernels_of, presolve

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 7, 8, 9, 16, 31, 32, 33, 40, 64, 255, 256, 257, 1000, 1023, 1024, 1025, 1056, 2047, 2048, 4096, 5003]


def trivial(i):   # a row without a live entry above the tolerance hashes its index
    return ((0xcbf29ce484222325 ^ i) * 0x100000001b3) & (2**64 - 1)


def oracle_hash(n, row_ptr, col_idx, values, row, keep_col, mode):
    at = slice(row_ptr[row], row_ptr[row + 1])
    one = np.array([0, row_ptr[row + 1] - row_ptr[row]], np.int32)   # the row by itself
    p = pyoracle.ptr
    h = pyoracle.lib().orc_row_hash(1, n, p(one), p(col_idx[at]), p(values[at]), 0, p(keep_col), mode)
    return trivial(row) if h == trivial(0) else h


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("mask", ["none", "half", "last", "nothing"])
@pytest.mark.parametrize("rows", [1, 200, 40_000])   # medium rows by fours, past 37,888 by 32
def test_row_hashes(mode, mask, rows):
    import torch
    rng = np.random.default_rng(mode)
    n = 6000
    lengths = np.array(LENGTHS + rng.integers(0, 80, 150).tolist() + rng.integers(900, 3000, 30).tolist())
    lengths = np.concatenate([lengths, np.full(rows, 9) + rng.integers(0, 3, rows)])
    lengths = lengths[rng.permutation(lengths.size)]
    m = lengths.size
    row_ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    col_idx = np.concatenate([np.sort(rng.choice(n, k, replace=False)) if k > 99 else np.unique(rng.integers(0, n, 2 * k))[:k] for k in lengths]).astype(np.int32)
    values = rng.standard_normal(col_idx.size)
    odd = rng.random(values.size)
    values[odd < 0.002] = np.inf
    values[(odd > 0.002) & (odd < 0.003)] = np.nan
    first = row_ptr[:-1][lengths > 0]
    values[first[::5]] = 1e-10   # a pivot at the tolerance
    keep_row = (rng.random(m) < 0.9).astype(np.uint8)
    keep_col = {"none": None, "half": rng.random(n) < 0.5, "last": np.arange(n) > n - 300,
                "nothing": np.zeros(n, bool)}[mask]
    keep_col = None if keep_col is None else keep_col.astype(np.uint8)
    dev = [to_device(row_ptr, np.int32), to_device(col_idx, np.int32), to_device(values, np.float64)]
    dk, dc = to_device(keep_row, np.uint8), None if keep_col is None else to_device(keep_col, np.uint8)
    out = torch.zeros(m, dtype=torch.int64, device="cuda")
    A = capi.Csr(m, n, int(col_idx.size), *(ptr(t) for t in dev))
    _raise(capi.load().gpp_parallel_row_hashes(C.byref(A), ptr(dk), ptr(dc), mode, ptr(out)))
    got = out.cpu().numpy().view(np.uint64)
    want = np.array([oracle_hash(n, row_ptr, col_idx, values, i, keep_col, mode) if keep_row[i] else i for i in range(m)],
                    dtype=np.uint64)
    assert np.array_equal(got, want), np.flatnonzero(got != want)


@pytest.mark.parametrize("m,per,aggregates", [(400, 200, True), (400, 20, False)])
def test_dense_matrices_take_the_order_free_form(m, per, aggregates):
    names = kernels_of(presolve(dense_lp(m, 2000, per, seed=per), capi.Params.defaults(enable_folding=0)))
    assert any("row_hash_kernel<true>" in k for k in names) == aggregates, names

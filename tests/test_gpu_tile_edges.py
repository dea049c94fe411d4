"""Single-pass compaction at the edges of its tiles (2,048 entries, 256 per
warp): entry counts one below, at and one above them, rows that start and end
there, runs of empty rows before, at and past the last entry; against numpy.
"""
import ctypes as C

import numpy as np
import pytest

from gpp_b200 import capi, lpgen
from gpp_b200.device import _d2h, _raise, ptr, to_device

pytestmark = pytest.mark.gpu


def model(layout, nnz, rng):
    if layout == "one row":
        lengths = [nnz]
    elif layout == "rows of 32":
        lengths = [32] * (nnz // 32) + ([nnz % 32] if nnz % 32 else [])
    elif layout == "edges":   # rows end at every warp's edge, empty rows around them
        lengths, left = [0, 0], nnz
        while left:
            lengths += [min(left, 256), 0, 0, 0]
            left -= min(left, 256)
    else:
        cuts = np.sort(rng.integers(0, nnz + 1, size=max(1, nnz // 7)))
        lengths = np.diff(np.concatenate([[0], cuts, [nnz]])).tolist() + [0] * 40
    row_ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    n = max(max(lengths), 50)
    col_idx = np.concatenate([np.sort(rng.choice(n, size=k, replace=False)) for k in lengths if k]).astype(np.int32)
    return len(lengths), n, row_ptr, col_idx, rng.standard_normal(nnz)


@pytest.mark.parametrize("layout", ["one row", "rows of 32", "edges", "random"])
@pytest.mark.parametrize("nnz", [1, 31, 255, 256, 257, 2047, 2048, 2049, 4096, 8 * 2048 + 1])
def test_compaction_at_tile_edges(nnz, layout):
    rng = np.random.default_rng(nnz)
    m, n, row_ptr, col_idx, values = model(layout, nnz, rng)
    for kept in (0.0, 0.5, 1.0):
        keep_r = (rng.random(m) < max(kept, 0.3)).astype(np.uint8)
        keep_c = (rng.random(n) < kept).astype(np.uint8)
        keep_r[0] = keep_c[0] = 1
        dev = [to_device(row_ptr, np.int32), to_device(col_idx, np.int32), to_device(values, np.float64)]
        A = capi.Csr(m, n, nnz, *(ptr(t) for t in dev))
        dkr, dkc = to_device(keep_r, np.uint8), to_device(keep_c, np.uint8)
        Ao, ATo = capi.Csr(), capi.Csr()
        _raise(capi.load().gpp_compact_and_transpose(C.byref(A), ptr(dkr), ptr(dkc), C.byref(Ao), C.byref(ATo)))
        rows = np.repeat(np.arange(m), np.diff(row_ptr))
        sel = keep_r[rows].astype(bool) & keep_c[col_idx].astype(bool)
        m2, n2 = int(keep_r.sum()), int(keep_c.sum())
        want = lpgen.coo_to_csr(m2, (np.cumsum(keep_r.astype(np.int64)) - 1)[rows[sel]],
                                (np.cumsum(keep_c.astype(np.int64)) - 1)[col_idx[sel]], values[sel])
        assert (Ao.rows, Ao.cols, Ao.nnz) == (m2, n2, int(sel.sum()))
        got = (_d2h(Ao.rowPtr, m2 + 1, np.int32), _d2h(Ao.colVal, Ao.nnz, np.int32), _d2h(Ao.nzVal, Ao.nnz, np.float64))
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
        for p in (Ao.rowPtr, Ao.colVal, Ao.nzVal, ATo.rowPtr, ATo.colVal, ATo.nzVal):
            capi.load().gpp_device_free(p)

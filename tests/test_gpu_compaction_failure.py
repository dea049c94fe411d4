"""A compaction whose allocations fail leaves its context fit for the next one: every
allocation fails in turn on a thread of its own (a fresh context, whose scratch still has
to grow), then the same call is made again; against numpy."""
import ctypes as C
import threading

import numpy as np
import pytest

from gpp_b200 import capi, lpgen
from gpp_b200.device import _d2h, _raise, ptr, to_device

pytestmark = pytest.mark.gpu


def compact(m, n, dev, dkr, dkc):
    A, Ao, ATo = capi.Csr(m, n, int(dev[2].numel()), *(ptr(t) for t in dev)), capi.Csr(), capi.Csr()
    code = capi.load().gpp_compact_and_transpose(C.byref(A), ptr(dkr), ptr(dkc), C.byref(Ao), C.byref(ATo))
    if code:
        return code, None
    got = [_d2h(Ao.rowPtr, Ao.rows + 1, np.int32), _d2h(Ao.colVal, Ao.nnz, np.int32), _d2h(Ao.nzVal, Ao.nnz, np.float64)]
    for p in (Ao.rowPtr, Ao.colVal, Ao.nzVal, ATo.rowPtr, ATo.colVal, ATo.nzVal):
        capi.load().gpp_device_free(p)
    return 0, got


@pytest.mark.parametrize("nnz", [3000, 9 << 20])   # kept row bits, and the call's own
def test_compaction_after_failed_allocations(nnz):
    rng = np.random.default_rng(nnz)
    length, n = 32, 4096
    m = nnz // length
    row_ptr = (np.arange(m + 1) * length).astype(np.int32)
    col_idx = ((np.arange(m * length) * 7) % n).astype(np.int32)   # any order within a row
    values = rng.standard_normal(m * length)
    keep_r, keep_c = (rng.random(m) < 0.6).astype(np.uint8), (rng.random(n) < 0.6).astype(np.uint8)
    sel = np.repeat(keep_r, length).astype(bool) & keep_c[col_idx].astype(bool)
    new_c = np.cumsum(keep_c, dtype=np.int64) - 1
    kept = sel.reshape(m, length).sum(axis=1)[keep_r.astype(bool)]
    want = [np.concatenate([[0], np.cumsum(kept)]).astype(np.int32), new_c[col_idx[sel]].astype(np.int32), values[sel]]
    dev = [to_device(row_ptr, np.int32), to_device(col_idx, np.int32), to_device(values, np.float64)]
    dkr, dkc = to_device(keep_r, np.uint8), to_device(keep_c, np.uint8)
    lib, seen = capi.load(), []

    def attempt(after):
        lib.gpp_inject_alloc_failure(after)
        try:
            code, _ = compact(m, n, dev, dkr, dkc)
        finally:
            lib.gpp_inject_alloc_failure(-1)
        again, got = compact(m, n, dev, dkr, dkc)
        seen.append((after, code, again, got is not None and all(np.array_equal(a, b) for a, b in zip(got, want))))

    failed = 0
    for after in range(24):
        t = threading.Thread(target=attempt, args=(after,))
        t.start()
        t.join()
        assert seen and seen[-1][0] == after and seen[-1][2] == 0 and seen[-1][3], seen[-1:]
        failed += seen[-1][1] != 0
    assert failed >= 4

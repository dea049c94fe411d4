"""Columns that are fixed one after the other, a segment of the record each: the restore
takes up to 64 segments a launch; the recovered point is the oracle's bit for bit."""
import numpy as np
import pytest

import pyoracle
from gpp_b200 import capi, device, lpgen

pytestmark = pytest.mark.gpu


def chain(n):
    """x_0 = 1 and x_k + x_{k+1} = k: a round of Cleanup fixes the next column; two more
    columns stay."""
    rows = np.concatenate([np.repeat(np.arange(n - 1), 2), [n - 1, n - 1]])
    cols = np.concatenate([np.column_stack([np.arange(n - 1), np.arange(1, n)]).ravel(), [n, n + 1]])
    p, i, v = lpgen.coo_to_csr(n, rows, cols, np.ones(rows.size))
    b = np.concatenate([np.arange(n - 1.0), [1.0]])
    l, u = np.full(n + 2, -1e6), np.full(n + 2, 1e6)
    l[0] = u[0] = 1.0
    return lpgen.HostLP(n, n + 2, p, i, v, np.ones(n + 2), b, b, l, u).ensure_transpose()


@pytest.mark.parametrize("n,launches", [(1, 1), (64, 1), (65, 2), (140, 3)])
def test_segments_of_fixed_columns(n, launches):
    import torch
    params = capi.params_with_rules(["infeasible_and_fixed_variables", "singleton_rows"], enable_folding=0, enable_startup=0)
    lp = chain(n)
    dlp = device.DeviceLp(lp)
    s = device.preprocess(dlp, params)
    try:
        assert len(device.Result(s).fixed_idx) == n and s.reduced_cols == 2
        point = [np.full(2, 0.5), np.ones(s.reduced_rows), np.ones(2)]
        got = device.postprocess(*(torch.from_numpy(v).cuda() for v in point), s, dlp)
        for a, b in zip(got, pyoracle.presolve(lp, params).postsolve(*point)):
            assert np.array_equal(a, b)
    finally:
        device.free_summary(s)
    lib = capi.load()
    lib.gpp_profile_enable(1)
    try:
        s = device.preprocess(dlp, params)
        device.postprocess(*(torch.from_numpy(v).cuda() for v in point), s, dlp)
        device.free_summary(s)
        assert {k: c for k, c, *_ in capi.profile_read()}["restore_fixed"] == launches
    finally:
        lib.gpp_profile_enable(0)

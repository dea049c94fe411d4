"""Replay of the postsolve tape by record groups against the oracle's serial
replay, bit for bit: tapes below and above the size that one block replays,
and points that sit on bounds, so that the row-implied bound changes act and
tie long runs of records together (points elsewhere leave most of them out).
"""
import numpy as np
import pytest

import pyoracle
from gpp_b200 import capi, device, lpgen

pytestmark = pytest.mark.gpu


def point(kind, l, u, rng):
    lo = np.where(np.isfinite(l), l, np.where(np.isfinite(u), u - 10.0, -10.0))
    hi = np.where(np.isfinite(u), u, lo + 20.0)
    if kind == "lower":
        return lo
    if kind == "upper":
        return hi
    x = np.where(rng.random(l.size) < 0.5, np.where(rng.random(l.size) < 0.5, lo, hi), lo + rng.random(l.size) * (hi - lo))
    if kind == "odd":
        x[rng.random(l.size) < 0.05] = np.nan
        x[rng.random(l.size) < 0.05] = np.inf
    return x


@pytest.mark.parametrize("kind", ["lower", "upper", "mixed", "odd"])
@pytest.mark.parametrize("workload,records", [("slack:400x1000", (1, 2048)), ("random:1500x3700", (1, 2048)),
                                              ("slack:2000x5000", (1, 2048)), ("slack:2100x5200", (2049, 1 << 30)),
                                              ("qap:4", (1, 2048)), ("qap:8", (2049, 1 << 30)),
                                              ("random:20000x50000", (2049, 1 << 30))])
def test_groups_replay_as_the_serial_tape(workload, records, kind):
    import torch
    lp = lpgen.workload(workload, seed=3)
    params = capi.Params.defaults(enable_folding=0)
    dlp = device.DeviceLp(lp)
    s = device.preprocess(dlp, params)
    try:
        gpu = device.Result(s)
        assert records[0] <= len(gpu.tape_types) <= records[1]
        rng = np.random.default_rng(5)
        xr = point(kind, gpu.l, gpu.u, rng)
        yr, zr = rng.standard_normal(s.reduced_rows), rng.standard_normal(s.reduced_cols)
        got = device.postprocess(*(torch.from_numpy(v).cuda() for v in (xr, yr, zr)), s, dlp)
        want = pyoracle.presolve(lp, params).postsolve(xr, yr, zr)
        for a, b in zip(got, want):
            assert np.array_equal(a, b, equal_nan=True)
    finally:
        device.free_summary(s)

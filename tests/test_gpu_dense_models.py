"""Dense models under the forms that suit sparse ones: which kernels they take, and
that the model and the recovered point are the oracle's bit for bit."""
import numpy as np
import pytest

import pyoracle
from gpp_b200 import capi, device, lpgen
from test_gpu_large_groups import compare

pytestmark = pytest.mark.gpu


def dense_lp(m, n, per, seed, slack=None):
    """m rows of `per` entries over n columns; with `slack`, equality rows with a singleton
    column each, bounded below ("bounded") or free with a cost ("free")."""
    rng = np.random.default_rng(seed)
    idx = np.concatenate([np.sort(rng.choice(n, per, replace=False)) for _ in range(m)])
    val = np.round(rng.uniform(-10.0, 10.0, m * per), 3) + 0.0005
    rows = np.repeat(np.arange(m), per)
    u = rng.uniform(1.0, 10.0, n)
    act = np.bincount(rows, weights=val * (rng.random(n) * u)[idx], minlength=m)
    l, c = np.zeros(n), rng.standard_normal(n)
    AL = np.where(rng.random(m) < 0.6, act - rng.uniform(0.5, 5.0, m), -np.inf)
    AU = np.where(rng.random(m) < 0.6, act + rng.uniform(0.5, 5.0, m), np.inf)
    if slack:
        rows, idx = np.concatenate([rows, np.arange(m)]), np.concatenate([idx, n + np.arange(m)])
        val = np.concatenate([val, np.where(rng.random(m) < 0.5, 1.0, -1.0)])
        l = np.concatenate([l, np.full(m, -np.inf if slack == "free" else 0.0)])
        u = np.concatenate([u, np.full(m, np.inf)])
        c = np.concatenate([c, rng.standard_normal(m) if slack == "free" else np.zeros(m)])
        AL, AU, n = act.copy(), act.copy(), n + m
    p, i, v = lpgen.coo_to_csr(m, rows, idx, val)
    return lpgen.HostLP(m, n, p, i, v, c, AL, AU, l, u).ensure_transpose()


def kernels_of(call):
    lib = capi.load()
    lib.gpp_profile_enable(1)
    try:
        call()
        return [name for name, *_ in capi.profile_read()]
    finally:
        lib.gpp_profile_enable(0)


def presolve(lp, params):
    dlp = device.DeviceLp(lp)
    return lambda: device.free_summary(device.preprocess(dlp, params))


@pytest.mark.parametrize("m,per,fused", [(320, 128, True), (321, 128, False), (1000, 300, False)])
def test_small_models_are_bounded_by_entries(m, per, fused):
    params = capi.Params.defaults(enable_folding=0)
    lp = dense_lp(m, 2000, per - 1, seed=m, slack="bounded")   # m * per entries: the line is at 40,960
    names = kernels_of(presolve(lp, params))
    assert any("probe_and_singleton_columns" in k for k in names) == fused, names
    assert fused or not any("inc_small" in k for k in names), names
    compare(lp, params)


@pytest.mark.parametrize("m,per,block", [(512, 300, True), (520, 40, True), (520, 300, False), (2040, 4, True), (2040, 60, False)])
def test_short_tapes_of_long_records(m, per, block):
    import torch
    params = capi.Params.defaults(enable_folding=0)
    lp = dense_lp(m, 2000, per, seed=m + per, slack="free")   # one substitution a row, of `per` entries
    dlp = device.DeviceLp(lp)
    s = device.preprocess(dlp, params)
    try:
        gpu = device.Result(s)
        assert len(gpu.tape_types) >= m and (block or len(gpu.tape_types) <= 2048)
        rng = np.random.default_rng(1)
        point = [rng.standard_normal(k) for k in (s.reduced_cols, s.reduced_rows, s.reduced_cols)]
        got = []
        names = kernels_of(lambda: got.extend(device.postprocess(*(torch.from_numpy(v).cuda() for v in point), s, dlp)))
        assert any("replay_block" in k for k in names) == block, (len(gpu.tape_types), names)
        for a, b in zip(got, pyoracle.presolve(lp, params).postsolve(*point)):
            assert np.array_equal(a, b)
    finally:
        device.free_summary(s)


@pytest.mark.parametrize("n", [1200, 9000])   # the fused refresh, and the launches
@pytest.mark.parametrize("seed", range(3))
def test_statistics_after_long_rows_and_columns_go(n, seed):
    """Rows without sides and columns with equal bounds go, of lengths around the rounds of a
    lane group (8, 32) and of a warp (65, 128); what then has one entry or none is found by
    the statistics that are left."""
    rng = np.random.default_rng(seed)
    lengths = [1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 66, 127, 128, 129, 193, 600, 1000]
    base = lpgen.random_lp(n // 3, n, seed, slack_frac=0.2)
    m, n, k = base.m, base.n, len(lengths)
    rows, cols = [np.repeat(np.arange(m), np.diff(base.row_ptr))], [base.col_idx]
    vals = [base.values]
    for i, length in enumerate(lengths):   # free rows, then fixed columns over the others' rows
        rows.append(np.full(length, m + i)); cols.append(np.sort(rng.choice(n, length, replace=False)))
        size = min(length, m)
        rows.append(np.sort(rng.choice(m, size, replace=False))); cols.append(np.full(size, n + i))
        vals += [rng.uniform(1.0, 2.0, length), rng.uniform(-2.0, 2.0, size)]
    p, i, v = lpgen.coo_to_csr(m + k, *(np.concatenate(a) for a in (rows, cols, vals)))
    lp = lpgen.HostLP(m + k, n + k, p, i, v, np.concatenate([base.c, rng.standard_normal(k)]),
                      np.concatenate([base.AL, np.full(k, -np.inf)]), np.concatenate([base.AU, np.full(k, np.inf)]),
                      np.concatenate([base.l, np.zeros(k)]), np.concatenate([base.u, np.zeros(k)])).ensure_transpose()
    assert (max(lp.m, lp.n) <= 8192 and lp.nnz <= 40960) == (n < 5000)
    compare(lp, capi.Params.defaults(enable_folding=0))

"""Sorts of few pairs, which compare each pair with all others, around the number at
which the passes take over (48 for each window of eight bits that varies), against
numpy's stable sort: equal keys among them, and keys that differ in the top bit."""
import ctypes as C

import numpy as np
import pytest

from gpp_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("windows", [1, 2, 5, 8])
@pytest.mark.parametrize("distinct", [3, 40, 1 << 62])
def test_small_sorts(windows, distinct):
    import torch
    line = 48 * windows
    for n in (2, 3, 31, 32, 33, line - 1, line, line + 1):
        rng = np.random.default_rng(n)
        pool = rng.integers(0, 1 << 64, size=min(distinct, n), dtype=np.uint64)
        keys = rng.choice(pool, n) & np.uint64((1 << 8 * windows) - 1)
        if windows == 8:
            keys[::5] |= np.uint64(1 << 63)
        vals = rng.permutation(n).astype(np.int32)
        k, v = torch.from_numpy(keys.view(np.int64)).cuda(), torch.from_numpy(vals).cuda()
        capi.check(capi.load().gpp_sort_pairs(C.c_void_p(k.data_ptr()), C.c_void_p(v.data_ptr()), n))
        order = np.argsort(keys, kind="stable")
        assert np.array_equal(k.cpu().numpy().view(np.uint64), keys[order]) and np.array_equal(v.cpu().numpy(), vals[order])

"""Sorts of more pairs than one block takes, whose keys vary in a few bytes only: the
passes of the others are left out, an odd or even number stays, none at all for equal
keys; runs of equal keys (one count for a warp) of lengths around 32 and 128; against
numpy's stable sort."""
import ctypes as C

import numpy as np
import pytest

from gpp_b200 import capi

pytestmark = pytest.mark.gpu

MASKS = [0, 0xFF, 0xFF << 56, 0xFF00FF, 0xFF << 24 | 0xFF << 40, 0x7 << 13, 0xFFFFFF << 20, (1 << 64) - 1]


@pytest.mark.parametrize("mask", MASKS, ids=hex)
@pytest.mark.parametrize("n", [8193, 65_537 + 31, (1 << 20) + 4097])
@pytest.mark.parametrize("run", [1, 31, 32, 33, 128, 5000])
def test_few_varying_bytes(n, mask, run):
    import torch
    rng = np.random.default_rng(run)
    runs = rng.integers(0, 1 << 64, size=n // run + 1, dtype=np.uint64) & np.uint64(mask)
    keys = (np.repeat(runs, run)[:n]) | (np.uint64(0x5A5A5A5A5A5A5A5A) & ~np.uint64(mask))
    vals = rng.permutation(n).astype(np.int32)
    k, v = torch.from_numpy(keys.view(np.int64)).cuda(), torch.from_numpy(vals).cuda()
    capi.check(capi.load().gpp_sort_pairs(C.c_void_p(k.data_ptr()), C.c_void_p(v.data_ptr()), n))
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(k.cpu().numpy().view(np.uint64), keys[order]) and np.array_equal(v.cpu().numpy(), vals[order])

"""The one-launch-per-pass radix sort at the sizes where its paths and tiles
change, against numpy's stable sort: one block up to 8,192 pairs, tiles of
2,048 pairs below 2^20 and of 4,096 from there; keys whose digits are all
equal (skipped passes, an odd number of passes left), ascending, descending."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [2, 31, 1024, 1025, 8191, 8192, 8193, 10240, 65537, (1 << 20) - 1, 1 << 20, (1 << 20) + 4097]


def make_keys(kind, rng, n):
    if kind == "random":
        return rng.integers(0, 2**64, size=n, dtype=np.uint64)
    if kind == "one digit":
        return (rng.integers(0, 256, size=n, dtype=np.uint64) << np.uint64(24)) | np.uint64(0x5500000000000033)
    if kind == "three digits":
        return rng.integers(0, 1 << 20, size=n, dtype=np.uint64) << np.uint64(40)
    if kind == "equal":
        return np.full(n, 0xFEDCBA9876543210, dtype=np.uint64)
    if kind == "skewed":   # most keys in one digit of every pass
        keys = np.zeros(n, dtype=np.uint64)
        few = rng.random(n) < 0.01
        keys[few] = rng.integers(0, 2**64, size=int(few.sum()), dtype=np.uint64)
        return keys
    return np.arange(n, dtype=np.uint64)[::-1].copy()


@pytest.mark.parametrize("kind", ["random", "one digit", "three digits", "equal", "skewed", "descending"])
@pytest.mark.parametrize("n", SIZES)
def test_sort_matches_numpy(n, kind):
    import torch
    from gpp_b200 import capi
    rng = np.random.default_rng(n)
    keys = make_keys(kind, rng, n)
    vals = rng.permutation(n).astype(np.int32)
    dk, dv = torch.from_numpy(keys.view(np.int64)).cuda(), torch.from_numpy(vals).cuda()
    capi.check(capi.load().gpp_sort_pairs(C.c_void_p(dk.data_ptr()), C.c_void_p(dv.data_ptr()), n))
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(dk.cpu().numpy().view(np.uint64), keys[order])
    assert np.array_equal(dv.cpu().numpy(), vals[order])

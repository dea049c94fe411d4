"""A sort whose tiles stop waiting for their predecessors' counts: the call returns an
error, and what it leaves are zeros, which kernels launched before the host has seen
the error can use as indices.  The next sort is right."""
import ctypes as C

import numpy as np
import pytest

from gpp_b200 import capi

pytestmark = pytest.mark.gpu

GPP_ERR_CUDA = 1


@pytest.mark.parametrize("n", [300_001, 3_000_001])   # tiles of 2,048 and of 4,096 pairs
def test_expired_wait_leaves_zeros(n):
    import torch
    lib = capi.load()
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 2**63, size=n, dtype=np.int64)
    vals = np.arange(1, n + 1, dtype=np.int32)

    def sort():
        k, v = torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda()
        return lib.gpp_sort_pairs(C.c_void_p(k.data_ptr()), C.c_void_p(v.data_ptr()), n), k, v

    expired = 0
    try:
        lib.gpp_inject_sort_wait_limit(1)   # gives up where the first look finds nothing
        for _ in range(20):
            status, k, v = sort()
            if status:
                assert status == GPP_ERR_CUDA and b"ran out" in lib.gpp_last_error()
                assert not k.any() and not v.any()
                expired += 1
    finally:
        lib.gpp_inject_sort_wait_limit(0)
    assert expired
    status, k, v = sort()
    assert status == 0, lib.gpp_last_error()
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(k.cpu().numpy(), keys[order]) and np.array_equal(v.cpu().numpy(), vals[order])

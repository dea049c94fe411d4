"""A presolve whose allocation fails leaves the thread's kept row schedules fit for the
next call.  They grow with the model, so every model here is larger than the one
before; its n-th allocation fails, then the same model is presolved undisturbed and
must reduce as on a thread that saw no failure."""
import ctypes as C
import threading

import pytest

from gpp_b200 import capi, lpgen

pytestmark = pytest.mark.gpu


def key(s):
    return (s.reduced_rows, s.reduced_cols, s.reduced_nnz, s.iterations, s.obj_constant_delta)


def test_growth_after_failed_allocations():
    from gpp_b200 import device
    lib = capi.load()
    params = capi.Params.defaults()
    models = [device.DeviceLp(lpgen.random_lp(300 + 10 * k, 750 + 25 * k, seed=k)) for k in range(110)]
    got, failed = [], []

    def disturbed():
        for after, dlp in enumerate(models):
            s = capi.Summary()
            lib.gpp_inject_alloc_failure(after)
            try:
                failed.append(lib.gpp_preprocess(C.byref(dlp.struct()), C.byref(params), C.byref(s)) != 0)
            finally:
                lib.gpp_inject_alloc_failure(-1)
            lib.gpp_free_summary(C.byref(s))
            s = device.preprocess(dlp, params)
            got.append(key(s))
            device.free_summary(s)

    t = threading.Thread(target=disturbed)
    t.start()
    t.join()
    want = []
    for dlp in models:
        s = device.preprocess(dlp, params)
        want.append(key(s))
        device.free_summary(s)
    assert sum(failed) >= 100
    assert got == want

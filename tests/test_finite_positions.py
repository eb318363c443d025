"""Positions that are not finite are refused wherever they stand (checked eight values at a time, host only), and the
lists a batch returns are the caller's own."""
import ctypes

import numpy as np
import pytest

from interaxplugin import BatchContext, System, _capi
from interaxplugin import workloads as W


@pytest.mark.parametrize("n", [1, 2, 3, 5, 6, 8, 11])
def test_every_place_is_checked(n):
    L = _capi.lib()
    req = ctypes.c_void_p()
    assert L.ix_request_create(n, None, ctypes.byref(req)) == _capi.IX_OK
    good = np.random.default_rng(n).normal(size=(n, 3)) * 1e150
    good.flat[0] = -0.0
    assert L.ix_request_set_state(req, _capi.ptr(good), None, None) == _capi.IX_OK
    for k in range(3 * n):
        for value in (np.nan, np.inf, -np.inf):
            x = good.copy()
            x.flat[k] = value
            assert L.ix_request_set_state(req, _capi.ptr(x), None, None) != _capi.IX_OK
            assert f"(particle {k // 3})".encode() in L.ix_last_error(req)
    L.ix_ctx_destroy(req)


def test_masses_follow_the_particles():
    system = System()
    system.addParticle(1.5)
    assert system._masses_array().tolist() == [1.5]
    system.addParticle(2.0)
    assert system._masses_array().tolist() == [1.5, 2.0]


@pytest.mark.gpu
def test_batch_results_are_the_callers():
    systems, positions = W.cluster_set(5, seed=3)
    batch = BatchContext(systems)
    e1, f1 = batch.compute(positions)
    kept = [f.copy() for f in f1]
    batch.compute([p * 1.02 for p in positions])
    assert all(np.array_equal(a, b) for a, b in zip(f1, kept))
    f1[0][:] = 0.0
    e2, f2 = batch.compute(positions)
    assert np.array_equal(e1, e2) and all(np.array_equal(a, b) for a, b in zip(kept, f2))

"""What handles keep between uses goes back to the device."""
import ctypes

import numpy as np
import pytest

import bhut_gb300 as bh
from bhut_gb300 import _lib, workloads
from bhut_gb300.api import _Handle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


def _used(L):
    used, reserved = ctypes.c_int64(), ctypes.c_int64()
    _lib.check(L.bhut_pool_usage(ctypes.byref(used), ctypes.byref(reserved)))
    return used.value, reserved.value


def test_trim_returns_idle_trees(engine_lib):
    import torch
    L = engine_lib
    _lib.check(L.bhut_pool_trim())
    before = _used(L)[0]
    pos, m = workloads.gaussian(5000, seed=1)
    first = bh.accelerations(pos, m, softening=0.01)
    handles = [_Handle(3, 32) for _ in range(3)]
    for h in handles:
        h.build(pos, m)
    for h in handles:
        h.close()
    _lib.check(L.bhut_pool_trim())
    torch.cuda.synchronize()
    assert _used(L)[0] <= before
    assert np.array_equal(bh.accelerations(pos, m, softening=0.01), first)

"""Trees kept for reuse after they are closed: the next one, of another size,
dimension, form or thread, starts from nothing but the memory."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import bhut_gb300 as bh
from bhut_gb300 import workloads
from bhut_gb300.api import morton_argsort

pytestmark = pytest.mark.gpu

CASES = [(n, dim, form) for n in (1, 40, 3000, 12_000) for dim in (3, 2)
         for form in ("fast", "exact", "fp32")]


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


def _solve(case):
    n, dim, form = case
    pos, m = workloads.gaussian(n, seed=n, dim=dim)
    return bh.accelerations(pos, m, dim=dim, softening=0.02, form=form)


def _on_own_stream(case):
    """The same on a stream given by the caller, which is never kept."""
    import torch
    n, dim, form = case
    pos, m = workloads.gaussian(n, seed=n, dim=dim)
    h = bh.api._Handle(dim, 32, stream=torch.cuda.Stream().cuda_stream)
    h.set_form(form)
    h.build(pos, m)
    out = np.empty((n, dim))
    h.accel_self(0.5, 0.02, 1.0, out)
    h.close()
    return out


@pytest.mark.parametrize("order", [1, 5, 7])
def test_reuse_leaves_nothing_behind(order):
    cases = [CASES[(k * order) % len(CASES)] for k in range(len(CASES))]
    for c in cases:
        assert np.array_equal(_solve(c), _on_own_stream(c)), c


def test_reuse_after_a_rejected_input():
    pos, m = workloads.gaussian(3000, seed=3000)
    ref = _solve((3000, 3, "fast"))
    bad = pos.copy()
    bad[7, 1] = np.nan
    for _ in range(3):
        with pytest.raises(ValueError):
            bh.accelerations(bad, m, softening=0.02)
        morton_argsort(pos[:100])
        assert np.array_equal(bh.accelerations(pos, m, softening=0.02), ref)


def test_threads():
    refs = {c: _solve(c) for c in CASES}
    jobs = [CASES[(7 * k) % len(CASES)] for k in range(72)]
    with ThreadPoolExecutor(8) as ex:
        for c, a in zip(jobs, ex.map(_solve, jobs)):
            assert np.array_equal(a, refs[c]), c

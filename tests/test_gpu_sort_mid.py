"""Inputs sorted in small tiles, with one or two launches a pass: the sizes at the edges
of the rule and of the tiles, spread and tied keys, both dimensions.  A stable
order is unique, so the permutation is compared exactly."""
import numpy as np
import pytest

import bhut_gb300 as bh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("kind", ["spread", "ties", "two clusters"])
@pytest.mark.parametrize("n", [4095, 4096, 4097, 8193, 8704, 8705, 10_000, 16_384, 16_385, 70_001,
                               319_999, 320_000, 320_001])
def test_stable_order(n, kind, dim):
    rng = np.random.default_rng(n + dim)
    pos = rng.uniform(-1.0, 1.0, (n, dim))
    if kind == "ties":
        pos = np.round(pos * 2.0) / 2.0
    elif kind == "two clusters":
        pos = pos * 1e-9 + rng.integers(0, 2, (n, 1))
    keys, perm = bh.morton_argsort(pos)
    own = np.empty_like(keys)
    own[perm] = keys
    assert np.array_equal(perm, np.argsort(own, kind="stable"))
    assert np.array_equal(keys, np.sort(own))
    # the keys themselves do not depend on how they are sorted
    box = np.vstack([pos.min(0), pos.max(0)])
    small = np.vstack([box, pos[:500]])
    k2, p2 = bh.morton_argsort(small)
    if np.array_equal(small.min(0), pos.min(0)) and np.array_equal(small.max(0), pos.max(0)):
        ref = np.empty_like(k2)
        ref[p2] = k2
        assert np.array_equal(ref[2:], own[:500])

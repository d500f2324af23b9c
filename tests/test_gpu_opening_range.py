"""Ratios whose squares leave the FP32 range: form fast opens what form exact
opens."""
import numpy as np
import pytest

import bhut_gb300 as bh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


@pytest.mark.parametrize("theta,size", [(0.0, 1e-20), (1e-30, 1e-20), (3e-23, 3e-23), (5e-23, 5e-23),
                                        (7e-23, 7e-23), (1e-22, 1e-22), (1.3e-22, 1.3e-22), (1.7e-22, 1.7e-22),
                                        (2.3e-22, 2.3e-22), (1e-20, 1e-20), (1e-15, 1e-15), (1e-8, 1e-8),
                                        (1e19, 1e-20), (1e30, 1e-20)])
def test_interaction_sets_at_extreme_theta(theta, size):
    """Points a multiple of `size` apart, seen from all over the box."""
    rng = np.random.default_rng(3)
    near = size * rng.uniform(-1.5, 1.5, (512, 3))
    corners = np.array(np.meshgrid([-1, 1], [-1, 1], [-1, 1]), float).reshape(3, -1).T
    pos = np.concatenate([near, corners, rng.uniform(-1, 1, (504, 3))]) * 0.99
    m = rng.uniform(0.5, 1.5, len(pos))
    st = {}
    for form in ("exact", "fast"):
        t = bh.Tree(pos, m, leaf_size=1, form=form).build()
        t.accelerations(theta=theta, softening=0.1)
        a = t._handle.stats()
        t.accelerations(pos[::-1] * 0.98, theta=theta, softening=0.1)
        st[form] = a, t._handle.stats()
        t.close()
    assert st["fast"] == st["exact"]

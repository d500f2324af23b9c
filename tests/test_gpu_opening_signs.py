"""Opening tests on squares keep the meaning of size / d >= theta: signs of
theta and of a TreeData's half sizes."""
import numpy as np
import pytest

import bhut_gb300 as bh
from bhut_gb300 import workloads
from bhut_gb300.api import compute_tree_statistics
from bhut_gb300.traverse import bh as walk

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("theta", [-1e-3, -0.5, -40.0])
def test_statistics_negative_theta_opens_all(dim, theta):
    pos, m = workloads.gaussian(500, seed=1, dim=dim)
    td = bh.build_tree(pos, m, leaf_size=8, backend="auto", dim=dim)
    got = compute_tree_statistics(td, pos[:50], theta)
    leaves = td.count[td.first_child == -1]
    assert got["avg_nodes_visited"] == len(td.mass)
    assert got["avg_monopoles_used"] == 0
    assert got["avg_particles_computed"] == np.sum(leaves - 1)


@pytest.mark.parametrize("half,opened", [(-1.0, False), (np.nan, False), (np.inf, True)])
def test_half_sizes_that_are_no_sizes(half, opened):
    pos, m = workloads.gaussian(300, seed=2)
    td = bh.build_tree(pos, m, leaf_size=300 // 2, backend="auto", dim=3)
    assert len(td.mass) == 3
    td.half_size[:] = half
    got = compute_tree_statistics(td, pos[:40], 0.5)
    assert got["avg_nodes_visited"] == (3 if opened else 1)
    for form, tol in (("exact", 1e-13), ("fast", 1e-10), ("fp32", 1e-5)):
        a = walk.barnes_hut_accelerations(td, pos, m, 0.05, 0.5, form=form)
        b = walk.barnes_hut_accelerations_targets(td, pos, m, pos[:40], 0.05, 0.5, form=form)
        if opened:
            d = pos[None, :, :] - pos[:, None, :]
            r2 = np.sum(d * d, axis=2) + 0.05 ** 2
            ref = np.sum(m[None, :, None] * d / r2[..., None] ** 1.5, axis=1)
        else:
            d = td.com[0] - pos
            ref = td.mass[0] * d / (np.sum(d * d, axis=1) + 0.05 ** 2)[:, None] ** 1.5
        assert np.linalg.norm(a - ref) <= tol * np.linalg.norm(ref), form
        assert np.linalg.norm(b - ref[:40]) <= tol * np.linalg.norm(ref[:40]), form

"""Nodes whose children are two leaves, taken in one visit: the leaf sizes where
the pair fits a block or does not, clusters that leave a child empty or with one
particle, a child without mass, and every form's counts against form "exact"."""
import numpy as np
import pytest

import bhut_gb300 as bh
from bhut_gb300 import batch, workloads
from conftest import rel_l2

pytestmark = pytest.mark.gpu

# form "fast": a pair within 2^-35 of FP64; "fp32": rsqrt 3 x 2^-22.9, five
# roundings of 2^-24, a plain sum of at most 32 terms, Kahan sums of runs.
# Half of the pairs' sizes may go into monopoles, which have the same bounds.
RTOL = {"fast": 2.0 ** -35, "fp32": 3 * 2.0 ** -22.9 + (5 + 32) * 2.0 ** -24}


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


def _solve(pos, m, form, leaf, dim, eps, targets=None, theta=0.5):
    tree = bh.Tree(pos, m, leaf_size=leaf, dim=dim, form=form).build()
    out = tree.accelerations(targets, theta=theta, softening=eps)
    stats = tree._handle.stats()
    tree.close()
    return out, stats


@pytest.mark.parametrize("eps", [0.05, 0.0])
@pytest.mark.parametrize("n,leaf,dim", [(2, 1, 3), (3, 1, 3), (33, 16, 3), (63, 31, 3), (64, 32, 3),
                                        (65, 32, 2), (66, 33, 3), (3000, 1, 2), (3001, 7, 3),
                                        (3000, 33, 3), (5001, 31, 3), (50_000, 32, 3)])
def test_counts_and_values(n, leaf, dim, eps):
    pos, _ = workloads.gaussian(n, seed=n, dim=dim)
    m = np.random.default_rng(n).uniform(0.5, 1.5, n)
    for targets in (None, pos[: min(n, 100)] * 1.5):
        ref, counts = _solve(pos, m, "exact", leaf, dim, eps, targets)
        fast, c = _solve(pos, m, "fast", leaf, dim, eps, targets)
        assert rel_l2(fast, ref) < RTOL["fast"]
        assert c == counts
        # theta 0: the FP32 opening test decides nothing
        ref, counts = _solve(pos, m, "exact", leaf, dim, eps, targets, 0.0) if n < 6000 else (0, 0)
        if n < 6000:
            f32, c = _solve(pos, m, "fp32", leaf, dim, eps, targets, 0.0)
            assert rel_l2(f32, ref) < RTOL["fp32"]
            assert c[:3] == counts[:3]


@pytest.mark.parametrize("form", ["fast", "fp32"])
@pytest.mark.parametrize("dead", ["zero", "cancelling"])
def test_child_without_mass(dead, form):
    n, leaf = 4000, 8
    pos, _ = workloads.gaussian(n, seed=5)
    m = np.random.default_rng(3).uniform(0.5, 1.5, n)
    side = pos[:, 0] > 0.1
    if dead == "zero":
        m[side] = 0.0
    else:
        m[side] = np.resize([1.0, -1.0], side.sum())
    # a mixed leaf that cancels is skipped by every form; theta 0 opens the rest
    ref, counts = _solve(pos, m, "exact", leaf, 3, 0.05, None, 0.0)
    out, c = _solve(pos, m, form, leaf, 3, 0.05, None, 0.0)
    assert c[:3] == counts[:3]
    assert rel_l2(out, ref) < 30 * RTOL[form]      # (signs: sums may lose a factor)


@pytest.mark.parametrize("form", ["fast", "fp32"])
@pytest.mark.parametrize("n", [1, 5, 200])
def test_no_mass_at_all(n, form):
    pos, _ = workloads.gaussian(n, seed=n)
    ref, counts = _solve(pos, np.zeros(n), "exact", 4, 3, 0.05)
    out, c = _solve(pos, np.zeros(n), form, 4, 3, 0.05)
    assert not out.any() and not ref.any()
    assert c == counts


@pytest.mark.parametrize("leaf", [1, 7, 16, 32])
@pytest.mark.parametrize("form,eps", [("fp32", 0.05), ("fp32", 0.0), ("fast", 0.05), ("fast", 0.0)])
def test_batch_equals_single(form, eps, leaf):
    systems = [workloads.gaussian(n, seed=n) for n in (700, 33, 1500)]
    pos, m, off = batch.concat_systems(systems)
    solver = batch.BatchedSolver(form=form, leaf_size=leaf, use_graph=False).load(pos, m, off)
    got = solver.solve(theta=0.5, softening=eps)
    counts = np.zeros(3, dtype=np.int64)
    for k, (p, mm) in enumerate(systems):
        one, c = _solve(p, mm, form, leaf, 3, eps)
        counts += c
        part = got[off[k]:off[k + 1]]
        if form == "fp32":
            assert np.array_equal(part, one)
        else:
            assert rel_l2(part, one) < RTOL[form]
    assert np.array_equal(solver.stats(), counts)
    solver.close()

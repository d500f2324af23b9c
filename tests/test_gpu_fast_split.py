"""Form "fast": distant leaves (biased sums, two sources to a row) and split
traversals (several warps per 32 targets), at the sizes where their edges are:
leaves with one source, odd counts and more than one block of 32, trees with
fewer leaves than a split has paths, part-filled target groups, targets inside
and outside the box."""
import numpy as np
import pytest

import bhut_gb300 as bh
from bhut_gb300 import workloads
from conftest import rel_l2

pytestmark = pytest.mark.gpu

# float-float against IEEE FP64: a pair is within 2^-35 (checked) or, softened,
# 2^-48 / (eps s) of itself; sums of one sign stay below it, sums of both signs
# lose what cancels (a factor of 30 is allowed)
RTOL, RTOL_SIGNS = 2.0 ** -35, 30 * 2.0 ** -35


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


def _masses(kind, n, rng):
    if kind == "equal":
        return np.full(n, 1.0 / n)
    m = rng.uniform(0.5, 1.5, n)
    return m * rng.choice([-1.0, 1.0], n) if kind == "signs" else m


def _both(pos, m, targets, dim, leaf, eps, theta=0.6):
    out = {}
    for form in ("fast", "exact"):
        t = bh.Tree(pos, m, leaf_size=leaf, dim=dim, form=form).build()
        out[form] = t.accelerations(targets, theta=theta, softening=eps), t._handle.stats()
        t.close()
    return out


@pytest.mark.parametrize("masses", ["equal", "uneven", "signs"])
@pytest.mark.parametrize("n,leaf,dim,eps", [
    (2, 1, 3, 0.05), (33, 32, 3, 0.05), (700, 1, 3, 0.05), (900, 2, 2, 0.05), (3001, 3, 3, 0.0),
    (5003, 31, 3, 0.05), (5003, 33, 2, 0.0), (9001, 70, 3, 0.05), (40_000, 16, 3, 0.0)])
def test_self_against_exact(n, leaf, dim, eps, masses):
    pos, _ = workloads.gaussian(n, seed=n + leaf, dim=dim)
    m = _masses(masses, n, np.random.default_rng(n))
    r = _both(pos, m, None, dim, leaf, eps)
    assert rel_l2(r["fast"][0], r["exact"][0]) < (RTOL_SIGNS if masses == "signs" else RTOL)
    assert r["fast"][1] == r["exact"][1]      # pairs, monopoles, visits: none lost or doubled


@pytest.mark.parametrize("eps", [0.0, 0.05])
@pytest.mark.parametrize("n,nt,scale", [(1, 1, 1.0), (40, 3, 1.0), (2000, 31, 0.5), (2000, 65, 4.0),
                                        (60_000, 1000, 0.7), (60_000, 20_000, 3.0)])
def test_targets_against_exact(n, nt, scale, eps):
    pos, m = workloads.plummer(n, seed=n)
    targets = scale * np.random.default_rng(nt).standard_normal((nt, 3))
    r = _both(pos, m, targets, 3, 32, eps)
    assert rel_l2(r["fast"][0], r["exact"][0]) < RTOL
    assert r["fast"][1] == r["exact"][1]


@pytest.mark.parametrize("nt", [1, 100, 5000])
def test_split_repeats_itself(nt):
    pos, m = workloads.plummer(30_000, seed=4)
    tree = bh.Tree(pos, m, form="fast").build()
    a = tree.accelerations(pos[:nt], softening=0.01)
    assert np.array_equal(a, tree.accelerations(pos[:nt], softening=0.01))
    tree.close()


@pytest.mark.parametrize("form", ["fast", "exact"])
@pytest.mark.parametrize("n,leaf", [(2, 1), (3, 1), (4, 1), (65, 32), (97, 32), (130, 32), (300, 8)])
def test_smallest_trees(oracle_mod, n, leaf, form):
    """Trees of two to a few leaves: paths that end above their last level."""
    pos, m = workloads.gaussian(n, seed=n)
    tree = bh.Tree(pos, m, leaf_size=leaf, form=form).build()
    a = tree.accelerations(theta=0.5, softening=0.05)
    ref = oracle_mod.accelerations(oracle_mod.build_tree(pos, m, leaf), pos, m, theta=0.5,
                                   softening=0.05)
    assert rel_l2(a, ref) < (RTOL if form == "fast" else 1e-13)
    tree.close()

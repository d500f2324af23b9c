"""The bottom-up pass over slot-ordered leaf lists: trees whose leaves lie at
two depths (holes in the list), lists shorter and longer than a merge group of
256 entries, and batches that mix all of them."""
import numpy as np
import pytest

import bhut_gb300 as bh
from bhut_gb300 import batch, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


# (particles, leaf size): one leaf; a hole beside the shallow leaf; lists of
# 256 and 512 entries, full and with holes; many groups
SHAPES = [(1, 1), (3, 1), (65, 32), (255, 1), (256, 1), (257, 1), (511, 2), (4096, 16),
          (4097, 16), (8193, 16), (50_001, 7)]


@pytest.mark.parametrize("n,leaf", SHAPES)
def test_tree_arrays_bit_exact(oracle_mod, n, leaf):
    pos, m = workloads.gaussian(n, seed=n + leaf)
    m = np.random.default_rng(n).uniform(0.5, 1.5, n)
    tree = bh.Tree(pos, m, leaf_size=leaf).build()
    td, ref = tree._tree, oracle_mod.build_tree(pos, m, leaf)
    tree.close()
    for f in ("first_child", "start", "count", "perm", "center", "half_size", "mass", "com"):
        assert np.array_equal(np.asarray(getattr(td, f)), np.asarray(getattr(ref, f))), f


@pytest.mark.parametrize("sizes", [[1, 2, 3, 65, 1], [4097, 1, 8193, 33, 40_000, 17],
                                   [16] * 7 + [100] + [16] * 300 + [5000]])
def test_batch_of_ragged_systems_equals_single_trees(sizes):
    systems = [workloads.plummer(n, seed=k) for k, n in enumerate(sizes)]
    got = batch.batched_accelerations(systems, theta=0.6, softening=0.02, leaf_size=16,
                                      form="fp32", multipole="quad")
    for k in {*range(min(8, len(sizes))), len(sizes) - 1}:
        p, m = systems[k]
        ref = bh.accelerations(p, m, theta=0.6, softening=0.02, leaf_size=16, form="fp32",
                               multipole="quad")
        assert np.array_equal(got[k], ref), k


@pytest.mark.parametrize("dim", [3, 2])
@pytest.mark.parametrize("n", [1, 2, 31, 1023, 1024, 1025, 2049, 4097, 8191, 8192, 8193])
def test_small_orders_equal_the_oracle(oracle_mod, n, dim):
    """Points ordered by one block (the smallest) and by passes: keys with many
    ties (a coarse lattice, and all points in one) and distinct ones."""
    rng = np.random.default_rng(n)
    for pos in (rng.standard_normal((n, dim)), rng.integers(0, 4, (n, dim)).astype(float),
                np.ones((n, dim))):
        m = rng.uniform(0.5, 1.5, n)
        td = bh.Tree(pos, m, leaf_size=16, dim=dim).build()._tree
        ref = oracle_mod.build_tree(pos, m, 16)
        for f in ("perm", "center", "half_size", "mass", "com"):
            assert np.array_equal(np.asarray(getattr(td, f)), np.asarray(getattr(ref, f))), f


@pytest.mark.parametrize("n,leaf", [(40, 64), (3000, 16), (20_000, 16)])
def test_refit_and_rebuild_rule(oracle_mod, n, leaf):
    """A refit within 1.1 x the root box keeps the order and the boxes; one
    particle beyond it along one axis rebuilds."""
    pos, m = workloads.gaussian(n, seed=n)
    tree = bh.Tree(pos, m, leaf_size=leaf).build()
    first = tree._tree
    tree.refit(pos * 1.05)
    td = tree._tree
    assert np.array_equal(td.perm, first.perm) and np.array_equal(td.center, first.center)
    at = pos[np.asarray(td.perm)] * 1.05
    for k in (0, len(td.mass) - 1):
        s, c = int(td.start[k]), int(td.count[k])
        w = m[np.asarray(td.perm)][s:s + c]
        assert np.allclose(td.com[k], (at[s:s + c] * w[:, None]).sum(0) / w.sum(), rtol=1e-12)
    far = pos.copy()
    far[n // 2, 1] = first.center[0, 1] + 1.1001 * first.half_size[0]
    tree.refit(far)
    ref = oracle_mod.build_tree(far, m, leaf)
    assert np.array_equal(np.asarray(tree._tree.perm), np.asarray(ref.perm))
    assert np.array_equal(np.asarray(tree._tree.center), np.asarray(ref.center))
    tree.close()

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

"""The bottom-up pass with one lane to a node (long leaf lists), against the
oracle bit for bit, on both sides of the rule that chooses it."""
import numpy as np
import pytest

import bhut_gb300 as bh
from bhut_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


# (particles, leaf size, dim): lists of 32,768 / 65,536 entries (3-D), 4,096 /
# 8,192 / 16,384 (2-D), with and without holes
@pytest.mark.parametrize("n,leaf,dim", [(32_768, 1, 3), (32_769, 1, 3), (65_536, 1, 3),
                                        (70_001, 2, 3), (4096, 1, 2), (4097, 1, 2),
                                        (16_384, 1, 2), (30_011, 3, 2)])
@pytest.mark.parametrize("masses", ["uneven", "some zero"])
def test_tree_arrays_bit_exact(oracle_mod, n, leaf, dim, masses):
    pos, _ = workloads.gaussian(n, seed=n + leaf, dim=dim)
    rng = np.random.default_rng(n)
    m = rng.uniform(0.5, 1.5, n)
    if masses == "some zero":
        m[pos[:, 0] > 0.7] = 0.0
    tree = bh.Tree(pos, m, leaf_size=leaf, dim=dim).build()
    td, ref = tree._tree, oracle_mod.build_tree(pos, m, leaf)
    for f in ("perm", "center", "half_size", "mass", "com"):
        assert np.array_equal(np.asarray(getattr(td, f)), np.asarray(getattr(ref, f))), f
    # a refit to the same positions sums the same numbers
    tree.refit(pos)
    again = tree._tree
    for f in ("perm", "center", "half_size", "mass", "com"):
        assert np.array_equal(np.asarray(getattr(again, f)), np.asarray(getattr(td, f))), f
    tree.close()

"""Trees of a few long leaves: the warps that share 32 targets share a leaf's
particles too (blocks of 64), each exactly once."""
import numpy as np
import pytest

import bhut_gb300 as bh
from bhut_gb300 import workloads
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


# form fast is held to 1e-10 relative L2 of FP64, and to its interaction counts
@pytest.mark.parametrize("dim,eps", [(3, 0.05), (3, 0.0), (2, 0.05), (2, 0.0)])
@pytest.mark.parametrize("n", [2, 33, 64, 65, 128, 129, 257, 511, 513, 1025, 3000])
@pytest.mark.parametrize("leaves", [1, 2, 3, 5])
def test_long_leaves_against_exact(leaves, n, dim, eps):
    leaf = -(-n // leaves)
    pos, m = workloads.gaussian(n, seed=n, dim=dim)
    m = m * np.random.default_rng(n).uniform(0.5, 1.5, n)
    targets = np.concatenate([pos[:70] * 0.97, pos[:1] * 40])
    got = {}
    for form in ("exact", "fast"):
        t = bh.Tree(pos, m, leaf_size=leaf, dim=dim, form=form).build()
        got[form] = []
        for tg in (None, targets, targets[:1], targets[:33]):
            a = t.accelerations(tg, theta=0.4, softening=eps)
            assert np.array_equal(a, t.accelerations(tg, theta=0.4, softening=eps))
            got[form].append((a, t._handle.stats()))
        t.close()
    for (a, sa), (b, sb) in zip(got["fast"], got["exact"]):
        assert rel_l2(a, b) <= 1e-10
        assert sa[1:] == sb[1:]
        assert sa[0] == sb[0] or eps == 0.0   # (form exact leaves out pairs at no distance)

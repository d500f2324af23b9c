"""A target's value in forms exact and fp32 depends on the tree alone: not on how
many targets a call has, nor on which."""
import numpy as np
import pytest

import bhut_gb300 as bh
from bhut_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


@pytest.mark.parametrize("form", ["exact", "fp32"])
@pytest.mark.parametrize("n,dim,leaf", [(1, 3, 32), (40, 2, 1), (500, 3, 8), (3000, 3, 32), (20_000, 2, 16),
                                        (70_000, 3, 32), (200_000, 3, 64)])
def test_targets_by_call_size(n, dim, leaf, form):
    pos, m = workloads.gaussian(n, seed=n, dim=dim)
    tree = bh.Tree(pos, m, leaf_size=leaf, dim=dim, form=form).build()
    rng = np.random.default_rng(0)
    t = np.concatenate([pos[rng.integers(0, n, 2000)] * 1.01, rng.uniform(-9, 9, (500, dim))])
    kw = dict(theta=0.6, softening=0.02)
    ref = tree.accelerations(t, **kw)
    for k in (1, 2, 31, 33, 500):
        sel = rng.permutation(len(t))[:k]
        assert np.array_equal(tree.accelerations(t[sel], **kw), ref[sel]), k
    more = np.concatenate([t, rng.normal(0, 2, (60_000 if n <= 20_000 else 3000, dim))])
    assert np.array_equal(tree.accelerations(more, **kw)[:len(t)], ref)
    parts = tree.accelerations_chunks([t[:7], t[7:600], t[600:]], **kw)
    assert np.array_equal(np.concatenate(parts), ref)
    tree.close()

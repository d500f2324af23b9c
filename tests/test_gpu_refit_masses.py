"""Refits that change the masses: the frame of the FP32 forms (the unit of
mass, the equal-mass path) follows the masses of the refit, not of the build."""
import numpy as np
import pytest

import bhut_gb300 as bh
from bhut_gb300 import workloads
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


def _masses(kind, n, seed):
    rng = np.random.default_rng(seed)
    return {"equal": np.full(n, 1.0 / n), "other": np.full(n, 3.0),
            "uneven": rng.uniform(0.5, 1.5, n), "huge": rng.uniform(0.5, 1.5, n) * 1e45,
            "signs": rng.choice([-1.0, 1.0], n) * rng.uniform(0.5, 1.5, n)}[kind]


def _values(tree, targets):
    got = {}
    for form, multipole in (("exact", "mono"), ("fast", "mono"), ("fp32", "mono"), ("fp32", "quad")):
        tree.set_form(form, multipole=multipole)
        got[form, multipole] = tree.accelerations(softening=0.05), tree.accelerations(targets, softening=0.05)
    tree.close()
    return got


# A tree built with the second masses and refitted with them has the same
# topology, box and moments, so every form must agree bit for bit.  Besides,
# form fast is held to 1e-10 relative L2 of FP64 and form fp32 to the rounding
# of its terms.
@pytest.mark.parametrize("only", [False, True])
@pytest.mark.parametrize("dim,n", [(3, 3000), (2, 700)])
@pytest.mark.parametrize("first,then", [("equal", "uneven"), ("uneven", "equal"), ("equal", "other"),
                                        ("equal", "huge"), ("huge", "uneven"), ("equal", "signs")])
def test_refit_with_other_masses(first, then, dim, n, only):
    pos, _ = workloads.gaussian(n, seed=5, dim=dim)
    moved = pos * 0.99
    m0, m1 = _masses(first, n, 1), _masses(then, n, 2)
    trees = []
    for m in (m0, m1):
        t = bh.Tree(pos, m, leaf_size=16, dim=dim).build()
        t.accelerations(softening=0.05)                 # copies of the first masses exist
        if only:
            t._handle.refit_only(moved, m1)
        else:
            t.refit(moved, m1)
        trees.append(t)
    got, same = (_values(t, pos[:200] * 1.05) for t in trees)
    for k in range(2):
        ref = got["exact", "mono"][k]
        assert rel_l2(got["fast", "mono"][k], ref) <= 1e-10
        assert rel_l2(got["fp32", "mono"][k], ref) <= 1e-5
        for form in got:
            assert np.array_equal(got[form][k], same[form][k]), form

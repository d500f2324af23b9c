"""Form "fp32": leaf blocks read two sources to a row, filled with stand-ins
that add exactly zero, at the block sizes where they are (one source, one row
short, a full block, more than one block), for targets inside and outside the
box.  theta 0 sums every pair, so no opening decision enters."""
import numpy as np
import pytest

import bhut_gb300 as bh
from bhut_gb300 import workloads
from conftest import rel_l2

pytestmark = pytest.mark.gpu

# a pair: rsqrt 3 x 2^-22.9 and five roundings of 2^-24; a block's plain sum of
# at most 32 terms: 32 x 2^-24; Kahan sums add nothing at this size
RTOL = 3 * 2.0 ** -22.9 + (5 + 32) * 2.0 ** -24


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


@pytest.mark.parametrize("eps", [0.05, 0.0])
@pytest.mark.parametrize("masses", ["equal", "uneven"])
@pytest.mark.parametrize("n,leaf,dim", [(1, 1, 3), (9, 1, 3), (33, 7, 3), (72, 9, 2), (128, 8, 3),
                                        (500, 16, 3), (500, 32, 2), (999, 70, 3)])
def test_against_exact(n, leaf, dim, masses, eps):
    pos, m = workloads.gaussian(n, seed=n + leaf, dim=dim)
    if masses == "uneven":
        m = np.random.default_rng(n).uniform(0.5, 1.5, n)
    rng = np.random.default_rng(leaf)
    for targets in (None, rng.standard_normal((50, dim)), 40.0 * rng.standard_normal((33, dim))):
        out = []
        for form in ("fp32", "exact"):
            t = bh.Tree(pos, m, leaf_size=leaf, dim=dim, form=form).build()
            out.append(t.accelerations(targets, theta=0.0, softening=eps))
            t.close()
        if n > 1 or targets is not None:
            assert rel_l2(*out) < RTOL
        else:
            assert not out[0].any()

"""Refits that keep the tree while particles leave its box: forms fast and fp32
stay as accurate as inside."""
import pytest

import bhut_gb300 as bh
from bhut_gb300 import workloads
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


@pytest.mark.parametrize("scale", [1.5, 100.0, 1e6])
def test_refit_far_beyond_the_box(scale):
    """refit_only keeps the tree wherever the particles go."""
    pos, m = workloads.gaussian(2000, seed=6)
    t = bh.Tree(pos, m, leaf_size=16).build()
    t.accelerations(softening=0.05)
    t._handle.refit_only(pos * scale, m)
    got = {}
    for form in ("exact", "fast", "fp32"):
        t.set_form(form)
        got[form] = (t.accelerations(softening=0.05),
                     t.accelerations(pos[:100] * scale, softening=0.05))
    t.close()
    for k in range(2):
        assert rel_l2(got["fast"][k], got["exact"][k]) <= 1e-10
        assert rel_l2(got["fp32"][k], got["exact"][k]) <= 1e-5

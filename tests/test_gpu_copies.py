"""The FP32 copies of particles and nodes, made in integers: coordinates where the
fixed-point form has its edges (on the grid, halfway between its points, tiny
offsets from the frame's centre, the centre itself) in boxes of any scale."""
import numpy as np
import pytest

import bhut_gb300 as bh
from conftest import rel_l2

pytestmark = pytest.mark.gpu

# form "fast": a pair within 2^-35; "fp32": rsqrt 3 x 2^-22.9, five roundings of
# 2^-24 and a plain sum of at most 32 terms
RTOL = {"fast": 2.0 ** -35, "fp32": 3 * 2.0 ** -22.9 + (5 + 32) * 2.0 ** -24}


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


def _points(kind, n, rng):
    u = rng.uniform(-0.5, 0.5, (n, 3))
    if kind == "grid":
        u = np.round(u * 2.0 ** 23) / 2.0 ** 23
    elif kind == "halfway":
        u = (np.round(u * 2.0 ** 23) + 0.5) / 2.0 ** 23 + rng.integers(-1, 2, (n, 3)) * 2.0 ** -48
    elif kind == "centre":
        u[2:] *= 2.0 ** -rng.integers(0, 45, (n - 2, 1)).astype(float)
        u[2] = 0.0
    u[0], u[1] = -0.5, 0.5          # the frame: centre 0, half size 0.5
    return u


@pytest.mark.parametrize("form", ["fast", "fp32"])
@pytest.mark.parametrize("scale", [1.0, 3.0, 2.0 ** -60, 1e40])
@pytest.mark.parametrize("kind", ["spread", "grid", "halfway", "centre"])
def test_against_exact(kind, scale, form):
    rng = np.random.default_rng(len(kind))
    pos = _points(kind, 700, rng) * scale
    m = rng.uniform(0.5, 1.5, 700)
    out = []
    for f in (form, "exact"):
        t = bh.Tree(pos, m, leaf_size=8, form=f).build()
        out.append(t.accelerations(theta=0.0, softening=0.02 * scale))
        t.close()
    assert rel_l2(*out) < RTOL[form]

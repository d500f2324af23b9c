"""Form exact down to the bit where a value is a single term, and close to
rounding where it is a sum."""
import numpy as np
import pytest

import bhut_gb300 as bh
from bhut_gb300 import workloads
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


# Targets far from a small tree accept its root: one monopole each, with the
# integer square root of its r^2 + eps^2 in it.
@pytest.mark.parametrize("dim", [3, 2])
@pytest.mark.parametrize("span,mass", [(4, 1.0), (60, 0.7), (160, 3.3e-60), (160, 1.7e60)])
@pytest.mark.parametrize("eps", [0.0, 0.01])
def test_monopoles_bit_exact(eps, span, mass, dim):
    rng = np.random.default_rng(span)
    pos = rng.uniform(-1, 1, (37, dim)) * 1e-6
    m = mass * rng.uniform(0.5, 1.5, 37)
    n = 100_000
    t = np.ldexp(rng.uniform(1.0, 2.0, (n, dim)), rng.integers(0, span + 1, (n, 1)))
    t *= rng.choice([-1.0, 1.0], (n, dim))
    t[-5000:, 1:] *= rng.integers(0, 2, (5000, dim - 1))
    bits = t.view(np.uint64)
    k = rng.integers(0, 52, (n // 4, dim)).astype(np.uint64)
    bits[:n // 4] &= ~((np.uint64(1) << k) - np.uint64(1))      # short mantissas: exact squares, ties
    bits[n // 4:n // 2] |= (np.uint64(1) << k) - np.uint64(1)
    tree = bh.Tree(pos, m, leaf_size=4, dim=dim, form="exact").build()
    got = tree.accelerations(t, theta=0.5, softening=eps, G=1.25)
    assert tree._handle.stats() == (0, n, n)
    root = tree._tree
    tree.close()
    d = root.com[0] - t
    r2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]
    if dim == 3:
        r2 = r2 + d[:, 2] * d[:, 2]
    r2 = r2 + eps * eps
    f = (1.25 * root.mass[0]) / (r2 * np.sqrt(r2))
    assert np.array_equal(got, f[:, None] * d)


# n terms summed with at most n roundings each relative to the sum of their
# magnitudes, in runs and in pairs: a few 1e-16 of the rms in practice; 1e-14 is the
# form's bar against the oracle.
@pytest.mark.parametrize("n,dim,leaf", [(500, 3, 8), (5000, 3, 32), (20_000, 2, 16), (20_000, 3, 32)])
def test_sums_against_oracle(oracle_mod, n, dim, leaf):
    pos, m = workloads.gaussian(n, seed=n, dim=dim)
    tree = bh.Tree(pos, m, leaf_size=leaf, dim=dim, form="exact").build()
    a, b = tree.accelerations(softening=0.02), tree.accelerations(pos[:999], softening=0.02)
    tree.close()
    ot = oracle_mod.build_tree(pos, m, leaf)
    ref = oracle_mod.accelerations(ot, pos, m, theta=0.5, softening=0.02, G=1.0)
    assert rel_l2(a, ref) <= 1e-14
    assert rel_l2(b, ref[:999]) <= 1e-14

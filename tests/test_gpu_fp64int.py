"""FP64 pair arithmetic on the integer pipes: correctly rounded, so a pair of
form "exact" and of the direct sum equals numpy's separately rounded
operations bit for bit, over the whole range of doubles and at its edges."""
import numpy as np
import pytest

import bhut_gb300 as bh
from bhut_gb300 import workloads
from bhut_gb300.api import direct_accelerations

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


def _pairs(targets, m, eps):
    """Accelerations by one source of mass m at the origin, G = 1."""
    with np.errstate(all="ignore"):
        d = 0.0 - targets
        r2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]
        if d.shape[1] == 3:
            r2 = r2 + d[:, 2] * d[:, 2]
        r2 = r2 + eps * eps
        ri = 1.0 / np.sqrt(r2)
        f = m * ((ri * ri) * ri)
        return np.where((r2 == 0.0)[:, None], 0.0, 0.0 + f[:, None] * d)


def _same(a, b):
    return np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("dim,eps,span", [(3, 0.0, 3), (3, 0.01, 40), (2, 0.0, 300), (3, 0.0, 1020),
                                          (3, 1e-160, 1070)])
def test_pairs_bit_exact(dim, eps, span):
    rng = np.random.default_rng(span)
    n = 200_000
    t = np.ldexp(rng.uniform(1.0, 2.0, (n, dim)), rng.integers(-span, span + 1, (n, dim)).clip(max=1022))
    t *= rng.choice([-1.0, 1.0], (n, dim))
    bits = t.view(np.uint64)
    k = rng.integers(0, 52, (n // 4, dim)).astype(np.uint64)
    bits[:n // 4] &= ~((np.uint64(1) << k) - np.uint64(1))      # short mantissas: squares, ties
    bits[n // 4:n // 2] |= (np.uint64(1) << k) - np.uint64(1)   # ... and runs of ones
    t[-1000:] *= rng.integers(0, 2, (1000, dim))                # zero components
    for m in (1.0, 0.7, -3e-200, 0.0):
        got = direct_accelerations(np.zeros((1, dim)), np.array([m]), softening=eps, targets=t)
        assert _same(got, _pairs(t, m, eps)), m


@pytest.mark.parametrize("n,dim,leaf", [(1, 3, 32), (2, 3, 1), (33, 2, 32), (1000, 3, 16),
                                        (5000, 3, 32), (20_000, 2, 16)])
def test_exact_split_against_oracle(oracle_mod, n, dim, leaf):
    """Self solves and targets of form "exact", several warps per 32 targets:
    the oracle's pair terms in another order of summation."""
    pos, m = workloads.gaussian(n, seed=n, dim=dim)
    tree = bh.Tree(pos, m, leaf_size=leaf, dim=dim, form="exact").build()
    a, b = tree.accelerations(softening=0.02), tree.accelerations(pos[:999], softening=0.02)
    assert np.array_equal(a, tree.accelerations(softening=0.02))
    tree.close()
    ot = oracle_mod.build_tree(pos, m, leaf)
    ref = oracle_mod.accelerations(ot, pos, m, theta=0.5, softening=0.02, G=1.0)
    scale = np.sqrt(np.mean(ref * ref)) or 1.0
    bound = 4 * n * 2.0 ** -53            # n additions a side, each within half an ulp of the sum
    assert np.max(np.abs(a - ref)) <= max(bound, 1e-15) * 50 * scale
    assert np.max(np.abs(b - ref[:999])) <= max(bound, 1e-15) * 50 * scale

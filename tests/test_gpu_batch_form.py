"""Batches whose form changes after their systems were loaded: the buffers
follow the form that solves, with and without captured solves."""
import numpy as np
import pytest

from bhut_gb300 import workloads
from bhut_gb300.batch import BatchedSolver, concat_systems

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("dim,leaf,sizes", [(3, 8, (1, 9, 700, 5000)), (2, 32, (300, 4000)),
                                            (3, 1, (40, 1000))])
def test_form_changes_after_load(dim, leaf, sizes, use_graph):
    systems = [workloads.gaussian(n, seed=n, dim=dim) for n in sizes]
    loaded = concat_systems(systems)
    kw = dict(theta=0.5, softening=0.02)
    ref = {}
    for form in ("fp32", "fast"):
        sv = BatchedSolver(dim=dim, leaf_size=leaf, form=form, use_graph=use_graph).load(*loaded)
        ref[form] = sv.solve(**kw)
        sv.close()
    sv = BatchedSolver(dim=dim, leaf_size=leaf, form="fp32", use_graph=use_graph).load(*loaded)
    for k, form in enumerate(("fp32", "fast", "fp32", "fast", "fast")):
        sv.configure(form=form, use_graph=use_graph)
        if k == 3:   # the same layout again, then larger and smaller ones, in the new form
            sv.load(*loaded)
        assert np.array_equal(sv.solve(**kw), ref[form]), (k, form)
    more = concat_systems(systems + [workloads.gaussian(6000, seed=1, dim=dim)])
    for part in (more, loaded):
        sv.configure(form="fp32", use_graph=use_graph)
        sv.load(*part)
        sv.solve(**kw)
        sv.configure(form="fast", use_graph=use_graph)
        got = sv.solve(**kw)
        assert np.array_equal(got[:len(ref["fast"])], ref["fast"])
    sv.close()

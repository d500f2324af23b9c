"""The end of a handle waits for its own stream only."""
import pytest

from bhut_gb300 import workloads
from bhut_gb300.api import _Handle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    yield


@pytest.mark.parametrize("caller", [True, False])
@pytest.mark.parametrize("n", [1000, 600_000])
def test_end_of_a_handle_leaves_other_streams_alone(n, caller):
    """600,000 particles: larger than the trees that are kept."""
    import torch
    mine, other = torch.cuda.Stream(), torch.cuda.Stream()
    pos, m = workloads.gaussian(n, seed=2)
    P, M = torch.as_tensor(pos).cuda(), torch.as_tensor(m).cuda()
    a = torch.randn(8192, 8192, device="cuda", dtype=torch.bfloat16)
    b = torch.empty_like(a)
    stream = mine.cuda_stream if caller else None

    def use():
        h = _Handle(3, 32, stream)
        h.build(P, M)
        return h
    use().close()
    torch.matmul(a, a, out=b)
    h = use()
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    with torch.cuda.stream(other):
        for _ in range(400):        # some 0.2 s
            torch.matmul(a, a, out=b)
        done.record()
    h.close()
    waited = done.query()
    torch.cuda.synchronize()
    assert not waited

"""When nearestK builds its cell index, and a captured call's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from ompl_gb300 import base as B  # noqa: E402

PI = np.pi


def _index(dim, size, wrap=True):
    rng = np.random.default_rng(dim)
    nn = B.NearestNeighborsGPU(B.WrapL2StateSpace(dim) if wrap else B.RealVectorStateSpace(dim, -PI, PI),
                               capacity=size + 100)
    nn.add(torch.as_tensor(rng.uniform(-PI, PI, size=(size, dim)), device="cuda"))
    return rng, nn


@pytest.mark.parametrize("dim,size,nq", [(2, 100_000, 1024), (3, 200_000, 1024), (5, 100_000, 1024),
                                         (6, 600_000, 512), (7, 200_000, 4096), (8, 100_000, 8192)])
def test_first_large_batch(dim, size, nq):
    """The first batch that is worth an index builds it, after every change of the set."""
    rng, nn = _index(dim, size)
    q = torch.as_tensor(rng.uniform(-PI, PI, size=(nq, dim)), device="cuda")
    for _ in range(2):
        n0 = B.launch_count()
        nn.nearestK(q, 10)
        first = B.launch_count() - n0
        n0 = B.launch_count()
        nn.nearestK(q, 10)
        again = B.launch_count() - n0
        assert first > again > 3  # a build, then the cell search alone
        nn.add(q[:1])


@pytest.mark.parametrize("prefix", [False, True])
@pytest.mark.parametrize("dim,wrap,nq", [(7, True, 4096), (3, False, 4096)])
def test_captured_before_any_build(dim, wrap, nq, prefix):
    """A captured call that would build the index: its replays, and direct calls made before and after them."""
    size = 200_000
    rng, nn = _index(dim, 1000, wrap)
    nn = B.NearestNeighborsGPU(nn.space, capacity=size)
    pts = torch.as_tensor(rng.uniform(-PI, PI, size=(size, dim)), device="cuda")
    q = torch.as_tensor(rng.uniform(-PI, PI, size=(nq, dim)), device="cuda")
    lim = torch.as_tensor(rng.integers(0, size + 1, size=nq), device="cuda") if prefix else None
    nn.add(pts[:1000])
    nn.nearestK(q, 10, prefix=lim)  # the call's scratch, on a set that needs no index
    nn.add(pts[1000:])
    nn.setPrecision("fp64")
    want = nn.nearestK(q, 10, prefix=lim)
    nn.setPrecision("fp32_guarded")
    x = q.clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = nn.nearestK(x, 10, prefix=lim)
    for _ in range(2):  # the first of them builds
        got = nn.nearestK(q, 10, prefix=lim)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    for _ in range(2):
        out[0].fill_(-7)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out[0], want[0]) and torch.equal(out[1], want[1])


def test_scratch_grown_in_a_capture():
    """A captured call that needs more scratch than any call before it: direct calls of its size before its first
    replay, and replays."""
    rng, nn = _index(7, 20_000)
    q = torch.as_tensor(rng.uniform(-PI, PI, size=(1024, 7)), device="cuda")
    nn.setPrecision("fp64")
    want = nn.nearestK(q, 10)
    nn.setPrecision("fp32_guarded")
    nn.nearestK(q[:8].contiguous(), 10)
    x = q.clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = nn.nearestK(x, 10)
    for _ in range(2):
        got = nn.nearestK(q, 10)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out[0], want[0]) and torch.equal(out[1], want[1])

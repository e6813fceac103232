"""One index searched from several streams and threads at once, the first of the calls building its cell index: the
results of the exact FP64 scan."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from ompl_gb300 import base as B  # noqa: E402

PI = np.pi


def _setup(space, dim, size, sizes):
    rng = np.random.default_rng(dim)
    nn = B.NearestNeighborsGPU(space, capacity=size + 8)
    pts = torch.as_tensor(rng.uniform(-PI, PI, size=(size, dim)), device="cuda")
    nn.add(pts)
    qs = [torch.as_tensor(rng.uniform(-PI, PI, size=(n, dim)), device="cuda") for n in sizes]
    return nn, qs, _scan(nn, qs)


def _scan(nn, qs):
    nn.setPrecision("fp64")
    want = [nn.nearestK(q, 10) for q in qs]
    nn.setPrecision("fp32_guarded")
    torch.cuda.synchronize()
    return want


CASES = [("wrap", 7, 200_000), ("rv", 3, 200_000), ("chain", 10, 200_000)]


def _space(kind, dim):
    if kind == "chain":
        return B.KinematicChainSpace(dim, 0.1)
    return B.WrapL2StateSpace(dim) if kind == "wrap" else B.RealVectorStateSpace(dim, -PI, PI)


@pytest.mark.parametrize("kind,dim,size", CASES)
def test_streams(kind, dim, size):
    """Nothing orders the calls: the first builds, and the others search it from other streams."""
    nn, qs, want = _setup(_space(kind, dim), dim, size, [4096, 5000, 4500, 64, 6000, 300])
    streams = [torch.cuda.Stream() for _ in range(3)]
    for rep in range(3):
        if rep:  # the index is to be built again
            nn.add(qs[rep][:1])
            want = _scan(nn, qs)
        got = []
        for i, q in enumerate(qs):
            with torch.cuda.stream(streams[i % 3]):
                got.append(nn.nearestK(q, 10))
        torch.cuda.synchronize()
        for g, w in zip(got, want):
            assert torch.equal(g[0], w[0]) and torch.equal(g[1], w[1])


def test_threads():
    """Device batches and host rows, large and small, from four threads on streams of their own."""
    sizes = [4096, 1, 700, 5000, 33, 4500, 200, 6000] * 3
    nn, qs, want = _setup(_space("wrap", 7), 7, 200_000, sizes)
    want = [(i.cpu().numpy(), d.cpu().numpy()) for i, d in want]
    rows = [q.cpu().numpy() for q in qs]
    got, bad = {}, []

    def work(t):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for i in range(t, len(qs), 4):
                    if i % 3:
                        idx, dist = nn.nearestK(qs[i], 10)
                        stream.synchronize()
                        got[i] = (idx.cpu().numpy(), dist.cpu().numpy())
                    else:
                        got[i] = nn.nearestK(rows[i], 10)
        except Exception as e:  # reported below
            bad.append(e)

    ts = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
    for i, w in enumerate(want):
        assert np.array_equal(got[i][0], w[0]) and np.array_equal(got[i][1], w[1]), i

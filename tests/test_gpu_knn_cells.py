"""nearestK's cell search over large RealVector / wrapped indexes: the keys and FP64 distances of the exact FP64
scan, bit for bit, over dimensions, list lengths and prefix limits, for uniform, clustered, repeated, removed and
out-of-bounds elements."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from ompl_gb300 import base as B  # noqa: E402

PI = np.pi
N, NQ = 100_003, 4099  # 4.1e8 pairs: above the cell search's start in every dimension


def _space(kind, dim):
    return B.WrapL2StateSpace(dim) if kind == "wrap" else B.RealVectorStateSpace(dim, -PI, PI)


def _both(nn, q, k, prefix=None):
    out = []
    for p in ("fp64", "fp32_guarded"):
        nn.setPrecision(p)
        out.append(nn.nearestK(q, k, prefix=prefix))
    (i0, d0), (i1, d1) = out
    assert torch.equal(i0, i1)
    assert torch.equal(d0.view(torch.int64), d1.view(torch.int64))


def _index(kind, dim, pts):
    nn = B.NearestNeighborsGPU(_space(kind, dim), capacity=2 * len(pts))
    nn.add(torch.as_tensor(pts, device="cuda"))
    _warm(nn, dim)
    return nn


def _warm(nn, dim):
    """Enough pairs for the index to be built (results checked below come from it)."""
    q = torch.zeros((NQ, dim), dtype=torch.float64, device="cuda")
    for _ in range(5):
        nn.nearestK(q, 1)


@pytest.mark.parametrize("kind,dim", [("rv", 1), ("rv", 2), ("rv", 3), ("rv", 5), ("rv", 8), ("wrap", 1), ("wrap", 3),
                                      ("wrap", 7), ("wrap", 8)])
def test_uniform(kind, dim):
    rng = np.random.default_rng(dim)
    nn = _index(kind, dim, rng.uniform(-PI, PI, size=(N, dim)))
    q = torch.as_tensor(rng.uniform(-PI, PI, size=(NQ, dim)), device="cuda")
    for k in (1, 12, 13, 41, 64):
        _both(nn, q, k)
    pre = torch.as_tensor(rng.integers(-5, N + 5, size=NQ), device="cuda")
    _both(nn, q, 10, pre)
    _both(nn, q, 10, torch.sort(pre).values)
    # after a change of the set, and with half of it removed
    nn.add(torch.as_tensor(rng.uniform(-PI, PI, size=(5000, dim)), device="cuda"))
    nn.setPrecision("fp32_guarded")
    _warm(nn, dim)
    _both(nn, q, 10)
    nn.remove(rng.choice(N, size=N // 2, replace=False))
    nn.setPrecision("fp32_guarded")
    _warm(nn, dim)
    _both(nn, q, 10)
    _both(nn, q, 10, pre)


@pytest.mark.parametrize("kind,dim", [("rv", 3), ("wrap", 7)])
def test_uneven_data(kind, dim):
    rng = np.random.default_rng(7)
    clusters = rng.uniform(-PI, PI, size=(20, dim))[rng.integers(0, 20, N)] + rng.normal(0, 0.02, size=(N, dim))
    same = rng.uniform(-PI, PI, size=(50, dim))[rng.integers(0, 50, N)]
    for pts in (np.clip(clusters, -PI, PI), same):
        nn = _index(kind, dim, pts)
        q = pts[rng.integers(0, N, NQ)] + rng.normal(0, 0.01, size=(NQ, dim)) * (rng.random((NQ, 1)) < 0.7)
        _both(nn, torch.as_tensor(np.clip(q, -PI, PI), device="cuda"), 10)


def test_outside_the_bounds():
    """Elements and queries a little outside a RealVector space's bounds lie in the outermost levels."""
    rng = np.random.default_rng(9)
    pts = rng.uniform(-1.3 * PI, 1.3 * PI, size=(N, 3))
    nn = _index("rv", 3, pts)
    _both(nn, torch.as_tensor(rng.uniform(-1.5 * PI, 1.5 * PI, size=(NQ, 3)), device="cuda"), 10)


def test_small_index():
    """The smallest index of the cell search, and the sizes of its lowest prefix level."""
    rng = np.random.default_rng(12)
    for size in (16_383, 16_384, 16_385):
        nn = _index("rv", 2, rng.uniform(-PI, PI, size=(size, 2)))
        q = torch.as_tensor(rng.uniform(-PI, PI, size=(NQ, 2)), device="cuda")
        _both(nn, q, 10)
        pre = torch.as_tensor(np.sort(rng.integers(0, size + 1, size=NQ)), device="cuda")
        _both(nn, q, 10, pre)
        nn.setPrecision("fp32_guarded")

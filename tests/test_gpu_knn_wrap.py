"""nearestK's cell search at the wrap of a wrapped space: the keys and FP64 distances of the exact FP64 scan, bit for
bit, where many elements lie on both sides of +-pi at spacings below and above a cell level's rounding margin, where
elements are exactly -pi or pi, and where elements and queries lie outside [-pi, pi]."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from ompl_gb300 import base as B  # noqa: E402

PI = np.pi
N, NQ = 100_003, 4099


def _both(dim, pts, q, k=10):
    nn = B.NearestNeighborsGPU(B.WrapL2StateSpace(dim), capacity=len(pts))
    nn.add(torch.as_tensor(pts, device="cuda"))
    q = torch.as_tensor(q, device="cuda")
    for _ in range(5):  # enough pairs for the cell index to be built
        nn.nearestK(q, 1)
    pre = torch.as_tensor(np.sort(np.random.default_rng(1).integers(0, len(pts) + 1, size=len(q))), device="cuda")
    for prefix in (None, pre):
        out = []
        for p in ("fp64", "fp32_guarded"):
            nn.setPrecision(p)
            out.append(nn.nearestK(q, k, prefix=prefix))
        (i0, d0), (i1, d1) = out
        assert torch.equal(i0, i1)
        assert torch.equal(d0.view(torch.int64), d1.view(torch.int64))


def _fold(x):
    return (x + PI) % (2 * PI) - PI


@pytest.mark.parametrize("sigma", [1e-6, 1e-5, 2e-4, 1e-3, 1e-2])
@pytest.mark.parametrize("dim", [1, 2, 3, 5, 7, 8])
def test_clusters_across_the_wrap(dim, sigma):
    rng = np.random.default_rng([dim, int(1e6 * sigma)])
    pts = rng.uniform(-PI, PI, size=(N, dim))
    near = rng.permutation(N)[:3000]
    pts[near] = _fold(PI + rng.normal(0, sigma, size=(3000, dim)))
    pts[near[:40]] = rng.choice([-PI, PI], size=(40, dim))
    q = rng.uniform(-PI, PI, size=(NQ, dim))
    q[:600] = _fold(PI + rng.normal(0, sigma, size=(600, dim)))
    q[:20] = rng.choice([-PI, PI], size=(20, dim))
    _both(dim, pts, q[rng.permutation(NQ)])


@pytest.mark.parametrize("dim", [1, 2, 3, 5, 7, 8])
def test_outside_the_range(dim):
    rng = np.random.default_rng(dim)
    pts = rng.uniform(-1.6 * PI, 1.6 * PI, size=(N, dim))
    q = rng.uniform(-1.6 * PI, 1.6 * PI, size=(NQ, dim))
    # an element two turns less a little away: the folded distance is that little, below zero
    pts[:500] = 1.2 * PI + rng.normal(0, 1e-3, size=(500, dim))
    q[:200] = -0.8 * PI + rng.normal(0, 1e-3, size=(200, dim))
    _both(dim, pts, q)


@pytest.mark.parametrize("space", [B.WrapL2StateSpace(3), B.RealVectorStateSpace(3, -PI, PI)])
def test_queries_that_are_not_finite(space):
    """They have no neighbours, the others in the batch theirs."""
    rng = np.random.default_rng(2)
    nn = B.NearestNeighborsGPU(space, capacity=N)
    nn.add(torch.as_tensor(rng.uniform(-PI, PI, size=(N, 3)), device="cuda"))
    q = torch.as_tensor(rng.uniform(-PI, PI, size=(NQ, 3)), device="cuda")
    want = nn.nearestK(q, 10)
    odd = torch.arange(0, NQ, 7, device="cuda")
    for value in (float("nan"), float("inf"), -float("inf")):
        x = q.clone()
        x[odd, 1] = value
        idx, dist = nn.nearestK(x, 10)
        assert bool((idx[odd] == -1).all()) and bool(torch.isinf(dist[odd]).all())
        fine = torch.ones(NQ, dtype=torch.bool, device="cuda")
        fine[odd] = False
        assert torch.equal(idx[fine], want[0][fine]) and torch.equal(dist[fine], want[1][fine])

"""nearestK's one-launch form (small batches and indexes): the keys and FP64 distances of the exact FP64
scan, bit for bit, at the edges of its groups, buckets and cluster splits, with removed elements, prefix
limits, repeated points and both layouts; and against the CPU oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from ompl_gb300 import base as B  # noqa: E402

PI = np.pi


def _space(kind, dim):
    if kind == "chain":
        return B.KinematicChainSpace(dim, 0.1)
    return B.WrapL2StateSpace(dim) if kind == "wrap" else B.RealVectorStateSpace(dim, -PI, PI)


def _both(nn, q, k, prefix=None, soa=False):
    out = []
    for p in ("fp64", "fp32_guarded"):
        nn.setPrecision(p)
        out.append(nn.nearestK(q, k, prefix=prefix, soa=soa))
    (i0, d0), (i1, d1) = out
    assert torch.equal(i0, i1)
    assert torch.equal(d0.view(torch.int64), d1.view(torch.int64))


# 128 / 2048 / 5120: fewest groups for K = 16, 64 and 160 buckets; 8192 a warp's rounds; 16384 and 49152
# the group lengths; 70,001 several cluster splits
SIZES = [1, 7, 127, 129, 255, 257, 2047, 2049, 5119, 8193, 16383, 49153, 70001]


@pytest.mark.parametrize("kind,dim", [("rv", 2), ("rv", 3), ("rv", 7), ("wrap", 4), ("wrap", 7), ("chain", 6),
                                      ("chain", 10)])
@pytest.mark.parametrize("size", SIZES)
def test_matches_exact_scan(kind, dim, size):
    rng = np.random.default_rng(size * 31 + dim)
    nn = B.NearestNeighborsGPU(_space(kind, dim), capacity=size + 5)
    nn.add(torch.as_tensor(rng.uniform(-PI, PI, size=(size, dim)), device="cuda"))
    for nq in (1, 63, 65, 257):
        q = torch.as_tensor(rng.uniform(-PI, PI, size=(nq, dim)), device="cuda")
        for k in (1, 12, 20) if kind == "chain" else (1, 12, 13, 41, 64):
            _both(nn, q, k)
    q = torch.as_tensor(rng.uniform(-PI, PI, size=(dim, 65)), device="cuda")
    _both(nn, q, 5, soa=True)
    pre = torch.as_tensor(rng.integers(-1, size + 2, size=65), device="cuda")
    _both(nn, q, 5, prefix=pre, soa=True)
    _both(nn, q, 5, prefix=torch.sort(pre).values, soa=True)
    nn.remove(rng.choice(size, size=(size + 1) // 2, replace=False))
    _both(nn, q, 10, soa=True)


@pytest.mark.parametrize("kind,dim", [("rv", 2), ("wrap", 7), ("chain", 10)])
def test_repeated_points(kind, dim):
    """Equal distances: more elements within the guard band than the candidate list holds."""
    rng = np.random.default_rng(5)
    base = rng.uniform(-PI, PI, size=(3, dim))
    pts = base[rng.integers(0, 3, size=4000)]
    nn = B.NearestNeighborsGPU(_space(kind, dim), capacity=4000)
    nn.add(torch.as_tensor(pts, device="cuda"))
    q = torch.as_tensor(np.vstack([base, rng.uniform(-PI, PI, size=(67, dim))]), device="cuda")
    _both(nn, q, 10)
    _both(nn, q[:3], 10)


def test_non_finite_queries():
    rng = np.random.default_rng(6)
    nn = B.NearestNeighborsGPU(_space("rv", 3), capacity=3000)
    nn.add(torch.as_tensor(rng.uniform(-PI, PI, size=(3000, 3)), device="cuda"))
    q = torch.as_tensor(rng.uniform(-PI, PI, size=(4, 3)), device="cuda")
    q[1, 0] = float("nan")
    q[2, 1] = float("inf")
    _both(nn, q, 4)


def test_matches_oracle():
    from oracle.oracle import Oracle, SpaceDesc
    rng = np.random.default_rng(9)
    port = Oracle.port()
    sd = SpaceDesc(3, 7, np.full(7, -PI), np.full(7, PI))
    pts = rng.uniform(-PI, PI, size=(30000, 7))
    q = rng.uniform(-PI, PI, size=(40, 7))
    ri, rd = port.knn(sd, pts, q, 10)
    nn = B.NearestNeighborsGPU(B.WrapL2StateSpace(7), capacity=30000)
    nn.add(pts)
    i, d = nn.nearestK(q, 10)
    assert np.array_equal(i, ri)
    assert np.array_equal(d.view(np.uint64), rd.view(np.uint64))

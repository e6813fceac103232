"""nearestR with FP32 distances and FP64 decisions near the radius: counts, keys and distances of the FP64
form, bit for bit, over sizes at the edges of its launch shapes, short and long segments (both sorts),
removed elements, elements and queries outside the bounds, repeated distances and odd radii."""
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


def _both(nn, q, r):
    out = []
    for p in ("fp64", "fp32_guarded"):
        nn.setPrecision(p)
        out.append(nn.nearestR(q, r))
    for a, b in zip(*out):
        assert np.array_equal(a.view(np.int64) if a.dtype == np.float64 else a,
                              b.view(np.int64) if b.dtype == np.float64 else b)
    return out[1]


@pytest.mark.parametrize("kind,dim,r", [("rv", 2, 0.4), ("rv", 3, 0.5), ("rv", 7, 2.0), ("wrap", 7, 2.0),
                                        ("chain", 6, 0.5), ("chain", 10, 0.9)])
@pytest.mark.parametrize("size", [1, 31, 257, 2049, 4100, 20011])
def test_matches_fp64(kind, dim, r, size):
    rng = np.random.default_rng(size + dim)
    nn = B.NearestNeighborsGPU(_space(kind, dim), capacity=size)
    pts = rng.uniform(-PI, PI, size=(size, dim))
    nn.add(torch.as_tensor(pts, device="cuda"))
    for nq in (1, 63, 64, 66):
        q = rng.uniform(-PI, PI, size=(nq, dim))
        _both(nn, q, r)
    # the radius on an element's own FP64 distance: decided in FP64
    nn.setPrecision("fp64")
    _, d = nn.nearestK(q[:1], min(size, 16))
    _both(nn, q, float(d[0, -1]))
    for odd in (0.0, -1.0, float("nan")) + ((float("inf"),) if size <= 2049 else ()):
        _both(nn, q[:3], odd)
    nn.remove(rng.choice(size, size=(size + 1) // 2, replace=False))
    _both(nn, q, r)


@pytest.mark.parametrize("nq", [2, 65])
def test_segment_lengths(nq):
    """Segments at both sides of the in-place sort's start, of repeated distances."""
    rng = np.random.default_rng(3)
    nn = B.NearestNeighborsGPU(_space("rv", 2), capacity=6000)
    for n in (1024, 1, 1023, 2500):  # 1024, 1025, 2048, 4548 elements, all within the radius
        p = rng.integers(-20, 21, size=(n, 2)) / 10.0
        nn.add(torch.as_tensor(p, device="cuda"))
        _both(nn, rng.integers(-20, 21, size=(nq, 2)) / 10.0, 10.0)


def test_outside_the_bounds():
    rng = np.random.default_rng(4)
    nn = B.NearestNeighborsGPU(_space("rv", 3), capacity=9000)
    nn.add(torch.as_tensor(rng.uniform(-PI, PI, size=(4000, 3)), device="cuda"))
    q = rng.uniform(-PI, PI, size=(66, 3))
    q[5, 1], q[6, 0], q[7, 2] = 1e9, float("nan"), float("inf")
    _both(nn, q, 1.5)
    far = rng.uniform(-1e8, 1e8, size=(4000, 3))
    nn.add(torch.as_tensor(far, device="cuda"))
    q[:4] = far[:4] + 0.5
    _both(nn, q, 1.0)
    _both(nn, q, 3e7)

"""nearestK's cell search in a RealVector space whose bounds fix a coordinate (low == high), with elements and queries
off that plane: the keys and FP64 distances of the exact FP64 scan."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from ompl_gb300 import base as B  # noqa: E402

N, NQ = 100_003, 4099


@pytest.mark.parametrize("flat", [0, 1, 2])
def test_fixed_coordinate(flat):
    rng = np.random.default_rng(flat)
    low, high = np.full(3, -3.0), np.full(3, 3.0)
    low[flat] = high[flat] = 1.0
    pts, q = rng.uniform(-3.0, 3.0, size=(N, 3)), rng.uniform(-3.0, 3.0, size=(NQ, 3))
    q[:1000, flat] = 1.0
    nn = B.NearestNeighborsGPU(B.RealVectorStateSpace(3, low, high), capacity=N)
    nn.add(torch.as_tensor(pts, device="cuda"))
    q = torch.as_tensor(q, device="cuda")
    for _ in range(5):  # enough pairs for the cell index to be built
        nn.nearestK(q, 1)
    out = []
    for p in ("fp64", "fp32_guarded"):
        nn.setPrecision(p)
        out.append(nn.nearestK(q, 10))
    (i0, d0), (i1, d1) = out
    assert torch.equal(i0, i1)
    assert torch.equal(d0.view(torch.int64), d1.view(torch.int64))

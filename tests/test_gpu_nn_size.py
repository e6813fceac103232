"""size() counts the present elements after any order of add, remove and clear."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from ompl_gb300 import base as B  # noqa: E402


def test_size():
    rng = np.random.default_rng(0)
    nn = B.NearestNeighborsGPU(B.RealVectorStateSpace(3, -1.0, 1.0), capacity=1000)
    pts = rng.uniform(-1, 1, size=(1000, 3))
    assert nn.size() == 0
    nn.add(pts[:100])
    assert nn.size() == 100
    nn.remove(np.arange(10))
    nn.add(pts[100:150])  # before any count of what is left
    assert nn.size() == 140
    nn.remove(np.array([20]))
    nn.remove(np.array([20, 21]))
    nn.add(pts[150:151])
    assert nn.size() == 139
    assert nn.nearestK(pts[:1], 64)[0].min() >= 0
    nn.clear()
    assert nn.size() == 0

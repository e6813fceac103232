"""Host-array arguments in calls that are refused and from several threads."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from ompl_gb300 import base as B  # noqa: E402
from ompl_gb300 import workloads as W  # noqa: E402

PI = np.pi


def _setup(n=4000):
    rng = np.random.default_rng(1)
    space = B.RealVectorStateSpace(7, -PI, PI)
    space.setLongestValidSegmentFraction(1.0 / 300)
    ck = B.DHSphereArmValidityChecker(space, W.dh_arm(np.random.default_rng(2)), W.sphere_world(rng, 1500))
    nn = B.NearestNeighborsGPU(space, capacity=n)
    nn.add(torch.as_tensor(rng.uniform(-PI, PI, size=(n, 7)), device="cuda"))
    torch.cuda.synchronize()
    return rng, ck, nn


def test_a_refused_call_uses_no_buffer():
    """A call that is refused while its stream has queued work leaves no copy behind it for the next call's buffer."""
    rng, _, nn = _setup()
    a, b = rng.uniform(-PI, PI, size=(100, 7)), rng.uniform(-PI, PI, size=(10, 7))
    want = nn.nearestK(a, 20)
    slow, quick = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(slow):
        torch.cuda._sleep(200_000_000)
        with pytest.raises(RuntimeError):
            nn.nearestK(b, 65)
    with torch.cuda.stream(quick):
        for _ in range(300):
            got = nn.nearestK(a, 20)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])

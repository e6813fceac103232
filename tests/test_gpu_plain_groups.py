"""The plain motion form with several edges a warp: ok, first invalid index and segment count of one-edge calls, where
the batch does not divide evenly and its edges' lengths differ."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from ompl_gb300 import base as B  # noqa: E402
from ompl_gb300 import capi  # noqa: E402
from ompl_gb300 import workloads as W  # noqa: E402


@pytest.mark.parametrize("n", [4863, 4864, 4865, 7297, 50_001, 80_000])  # about 2, 3, 20 and 32 edges a warp
@pytest.mark.parametrize("soa", [False, True])
def test_groups(n, soa):
    rng = np.random.default_rng(n)
    space = B.RealVectorStateSpace(2, 0.0, 1.0)
    space.setLongestValidSegmentFraction(1.0 / 400)
    ck = B.CirclesValidityChecker(space, W.circles_world(rng))
    a, b = rng.uniform(0, 1, size=(n, 2)), rng.uniform(0, 1, size=(n, 2))
    b[: n // 2] = a[: n // 2] + 0.002 * (b[: n // 2] - a[: n // 2])
    mv = B.DiscreteMotionValidator(ck)
    t = [torch.as_tensor(np.ascontiguousarray(x.T if soa else x), device="cuda") for x in (a, b)]
    r = mv.checkMotions(*t, schedule=capi.SCHEDULE_PLAIN, soa=soa)
    assert 0.1 < r["ok"].double().mean() < 0.9
    step = 2000  # below the batch size at which a warp takes a second edge
    for i in range(0, n, step):
        part = mv.checkMotions(torch.as_tensor(a[i:i + step], device="cuda"),
                               torch.as_tensor(b[i:i + step], device="cuda"), schedule=capi.SCHEDULE_PLAIN)
        for key in ("ok", "first_j", "nd"):
            assert torch.equal(r[key][i:i + step], part[key]), (key, i)

"""DH arm worlds whose obstacles lie in one dense cluster (more of them near every cell than a list holds): the
oracle's verdicts, with the clearance of a sparse world of the same extent around them."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from ompl_gb300 import base as B  # noqa: E402
from ompl_gb300 import workloads as W  # noqa: E402
from oracle.oracle import CheckerDesc, Oracle, SpaceDesc  # noqa: E402

PI = math.pi


@pytest.mark.parametrize("n", [2048, 2049, 20_000])  # around the list's room
@pytest.mark.parametrize("boxes", [False, True])
def test_cluster(n, boxes):
    rng = np.random.default_rng(n)
    dh = W.dh_arm(np.random.default_rng(2))
    world = rng.uniform(0.002, 0.01, size=(n, 6 if boxes else 4))
    world[:, :3] = np.array([0.5, 0.45, 0.4]) + rng.uniform(-0.1, 0.1, size=(n, 3))
    world[0, :3], world[1, :3] = 1.5, -1.5
    s1, u = rng.uniform(-PI, PI, size=(1500, 7)), rng.normal(size=(1500, 7))
    s2 = np.clip(s1 + u * np.exp(rng.uniform(np.log(0.01), np.log(2.0), size=(1500, 1))), -PI, PI)
    space = B.RealVectorStateSpace(7, -PI, PI)
    space.setLongestValidSegmentFraction(1.0 / 600)
    sd = SpaceDesc(0, 7, np.full(7, -PI), np.full(7, PI), lvs_fraction=1.0 / 600)
    cd = CheckerDesc(W.CHECK_DH_BOXES if boxes else W.CHECK_DH_SPHERES, world, dh, 8, 0.05)
    port = Oracle.port()
    port.set_threads(16)
    ref = port.check_motion(sd, cd, s1, s2, want_state=False, want_bisect=False)
    assert 20 < ref["ok"].sum() < 1480  # verdicts of both kinds
    ck = (B.DHBoxArmValidityChecker if boxes else B.DHSphereArmValidityChecker)(space, dh, world)
    mv = B.DiscreteMotionValidator(ck)
    for p in ("fp64", "fp32_guarded"):
        ck.setPrecision(p)
        r = mv.checkMotions(s1, s2)
        for key in ("ok", "first_j", "nd"):
            assert np.array_equal(r[key], ref[key]), (p, key)

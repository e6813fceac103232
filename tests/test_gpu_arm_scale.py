"""DH arm worlds in other units than metres: the oracle's verdicts in both precisions where FP32 positions are coarser
than a fixed margin, and clearance that proves as much as in metres."""
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


def _world(scale, boxes):
    rng = np.random.default_rng(8)
    dh = W.dh_arm(np.random.default_rng(2))
    dh[:, :2] *= scale
    return dh, (W.box_world(rng, 1500) if boxes else W.sphere_world(rng, 1500)) * scale


def _edges(n):
    rng = np.random.default_rng(n)
    s1, u = rng.uniform(-PI, PI, size=(n, 7)), rng.normal(size=(n, 7))
    return s1, np.clip(s1 + u * np.exp(rng.uniform(np.log(0.01), np.log(2.0), size=(n, 1))), -PI, PI)


def _checker(dh, world, rs, boxes, fraction):
    space = B.RealVectorStateSpace(len(dh), -PI, PI)
    space.setLongestValidSegmentFraction(fraction)
    cls = B.DHBoxArmValidityChecker if boxes else B.DHSphereArmValidityChecker
    return cls(space, dh, world, 8 if len(dh) > 1 else 1, rs)


def _oracle(dh, world, rs, boxes, fraction, s1, s2):
    d = len(dh)
    port = Oracle.port()
    port.set_threads(16)
    sd = SpaceDesc(0, d, np.full(d, -PI), np.full(d, PI), lvs_fraction=fraction)
    cd = CheckerDesc(W.CHECK_DH_BOXES if boxes else W.CHECK_DH_SPHERES, world, dh, 8 if d > 1 else 1, rs)
    return port.check_motion(sd, cd, s1, s2, want_state=False, want_bisect=False)


@pytest.mark.parametrize("scale", [1e-2, 30.0, 1e3, 1e6])
@pytest.mark.parametrize("boxes", [False, True])
def test_verdicts(scale, boxes):
    dh, world = _world(scale, boxes)
    s1, s2 = _edges(1500)
    ref = _oracle(dh, world, 0.05 * scale, boxes, 1.0 / 600, s1, s2)
    ck = _checker(dh, world, 0.05 * scale, boxes, 1.0 / 600)
    mv = B.DiscreteMotionValidator(ck)
    for p in ("fp64", "fp32_guarded"):
        ck.setPrecision(p)
        r = mv.checkMotions(s1, s2)
        for key in ("ok", "first_j", "nd"):
            assert np.array_equal(r[key], ref[key]), (p, key)
        assert np.array_equal(ck.isValid(s2[ref["ok"] != 0]), np.ones(int(ref["ok"].sum()), dtype=bool))


@pytest.mark.parametrize("boxes", [False, True])
def test_contact_below_the_fp32_spacing(boxes):
    """One link of a million units whose only sphere touches the obstacle by half a thousandth: in FP32 its centre
    lies past everything the obstacle can touch."""
    a = 1000000.032
    dh = np.array([[a, 0.0, 0.0]])
    x = 0.5 * a - 1.9995
    world = np.array([[x, 0.0, 0.0, 1.0, 1.0, 1.0]]) if boxes else np.array([[x, 0.0, 0.0, 1.0]])
    s = np.zeros((3, 1))
    ref = _oracle(dh, world, 1.0, boxes, 0.01, s, s)
    assert not ref["ok"].any()
    ck = _checker(dh, world, 1.0, boxes, 0.01)
    mv = B.DiscreteMotionValidator(ck)
    for p in ("fp64", "fp32_guarded"):
        ck.setPrecision(p)
        assert np.array_equal(mv.checkMotions(s, s)["ok"], ref["ok"]), p
        assert not ck.isValid(s).any(), p


@pytest.mark.parametrize("scale", [1e3, 1e5])
@pytest.mark.parametrize("boxes", [False, True])
def test_clearance_does_not_depend_on_the_unit(scale, boxes):
    s1, s2 = _edges(3000)
    evaluated = []
    for f in (1.0, scale):
        dh, world = _world(f, boxes)
        ck = _checker(dh, world, 0.05 * f, boxes, 1.0 / 2500)
        ck.setPrecision("fp32_guarded")
        B.DiscreteMotionValidator(ck).checkMotions(s1, s2)
        evaluated.append(ck.stats()["evaluated"])
    assert evaluated[1] <= 1.1 * evaluated[0]

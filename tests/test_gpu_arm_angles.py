"""DH arm states with angles far outside a turn, infinite ones and NaN."""
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
DH = W.dh_arm(np.random.default_rng(2))
WORLD = W.sphere_world(np.random.default_rng(5), 1500)


def _setup():
    space = B.RealVectorStateSpace(7, -PI, PI)
    space.setLongestValidSegmentFraction(1.0 / 100)
    sd = SpaceDesc(0, 7, np.full(7, -PI), np.full(7, PI), lvs_fraction=1.0 / 100)
    port = Oracle.port()
    port.set_threads(16)
    return (B.DHSphereArmValidityChecker(space, DH, WORLD), port, sd,
            CheckerDesc(W.CHECK_DH_SPHERES, WORLD, DH, 8, 0.05))


@pytest.mark.parametrize("size", [90.0, 96.0, 100.0, 5e5, 9.9e5, 1.1e6, 2e6, 1e9, 1e13, 1e15])
def test_far_angles(size):
    """Both precisions, whole states and edges of a few steps, against the oracle."""
    ck, port, sd, cd = _setup()
    rng = np.random.default_rng(int(size))
    s1 = rng.uniform(-1.0, 1.0, size=(600, 7))
    s1[:, rng.integers(0, 7, size=600)] *= size
    s1 = np.where(rng.random((600, 7)) < 0.5, s1, rng.uniform(-PI, PI, size=(600, 7)))
    s1[np.arange(600), rng.integers(0, 7, 600)] = size * rng.choice([-1.0, 1.0], size=600) * rng.uniform(0.98, 1.02, 600)
    s2 = s1 + rng.uniform(-0.3, 0.3, size=(600, 7))
    ref = port.check_motion(sd, cd, s1, s2, want_state=False, want_bisect=False)
    valid = np.asarray(port.is_valid(sd, cd, s1)).astype(bool)
    assert 0 < valid.sum() < 600
    mv = B.DiscreteMotionValidator(ck)
    for p in ("fp64", "fp32_guarded"):
        ck.setPrecision(p)
        assert np.array_equal(ck.isValid(s1), valid), p
        r = mv.checkMotions(s1, s2)
        for key in ("ok", "first_j", "nd"):
            assert np.array_equal(r[key], ref[key]), (p, key)


def test_infinite_and_nan():
    """The finite edges of a batch keep the oracle's results; an edge with an end that is not finite has one step,
    its second end, judged as isValid judges it."""
    ck, port, sd, cd = _setup()
    rng = np.random.default_rng(4)
    for n in (60, 900):  # both launch forms
        s1 = rng.uniform(-PI, PI, size=(n, 7))
        s2 = np.clip(s1 + rng.normal(0, 0.2, size=(n, 7)), -PI, PI)
        odd = np.arange(0, n, 5)
        for m, i in enumerate(odd):
            (s1 if m & 1 else s2)[i, m % 7] = (np.nan, np.inf, -np.inf)[m % 3]
        fine = np.setdiff1d(np.arange(n), odd)
        ref = port.check_motion(sd, cd, s1[fine], s2[fine], want_state=False, want_bisect=False)
        ck.setPrecision("fp64")
        end = ck.isValid(s2)
        mv = B.DiscreteMotionValidator(ck)
        for p in ("fp64", "fp32_guarded"):
            ck.setPrecision(p)
            r = mv.checkMotions(s1, s2)
            for key in ("ok", "first_j", "nd"):
                assert np.array_equal(r[key][fine], ref[key]), (p, key)
            assert np.array_equal(r["ok"][odd] != 0, end[odd]), p
            assert (r["nd"][odd] <= 1).all()

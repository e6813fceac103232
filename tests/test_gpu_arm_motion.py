"""DH arm motion checking by clearance: ok, first invalid index and segment count of the oracle's
state-by-state check, in both precisions, over batch sizes at the edges of its launch forms, both joint
spaces, arm and world shapes, and inputs that the clearance must not judge."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from ompl_gb300 import base as B  # noqa: E402
from ompl_gb300 import capi  # noqa: E402
from ompl_gb300 import workloads as W  # noqa: E402
from oracle.oracle import CheckerDesc, Oracle, SpaceDesc  # noqa: E402

PI = math.pi


@pytest.fixture(scope="module")
def port():
    p = Oracle.port()
    p.set_threads(16)
    return p


def _compare(port, kind, dh, world, spl, rs, s1, s2, fraction=1.0 / 600, boxes=False):
    d = dh.shape[0]
    space = B.WrapL2StateSpace(d) if kind == "wrap" else B.RealVectorStateSpace(d, -PI, PI)
    space.setLongestValidSegmentFraction(fraction)
    sd = SpaceDesc(3 if kind == "wrap" else 0, d, np.full(d, -PI), np.full(d, PI), lvs_fraction=fraction)
    cd = CheckerDesc(W.CHECK_DH_BOXES if boxes else W.CHECK_DH_SPHERES, world, dh, spl, rs)
    ref = port.check_motion(sd, cd, s1, s2, want_state=False, want_bisect=False)
    cls = B.DHBoxArmValidityChecker if boxes else B.DHSphereArmValidityChecker
    ck = cls(space, dh, world, spl, rs)
    mv = B.DiscreteMotionValidator(ck)
    for p in ("fp64", "fp32_guarded"):
        ck.setPrecision(p)
        for sch in (capi.SCHEDULE_PLAIN, capi.SCHEDULE_TILE, capi.SCHEDULE_AUTO):
            r = mv.checkMotions(s1, s2, schedule=sch)
            for key in ("ok", "first_j", "nd"):
                assert np.array_equal(r[key], ref[key]), (p, sch, key)
    return ref


def _edges(rng, n, d, kind):
    s1 = rng.uniform(-PI, PI, size=(n, d))
    u = rng.normal(size=(n, d))
    u *= np.exp(rng.uniform(np.log(0.01), np.log(5.0), size=(n, 1))) / np.linalg.norm(u, axis=1, keepdims=True)
    s2 = s1 + u
    s2 = np.clip(s2, -PI, PI) if kind != "wrap" else (s2 + PI) % (2 * PI) - PI
    return s1, s2


@pytest.mark.parametrize("kind", ["rv", "wrap"])
@pytest.mark.parametrize("n", [1, 31, 767, 768, 769, 3041, 12200])
def test_batch_sizes(port, kind, n):
    rng = np.random.default_rng(n)
    s1, s2 = _edges(rng, n, 7, kind)
    ref = _compare(port, kind, W.dh_arm(np.random.default_rng(2)), W.sphere_world(rng, 1500), 8, 0.05, s1, s2)
    if n > 100:
        assert 0.05 < ref["ok"].mean() < 0.95


@pytest.mark.parametrize("joints,spl", [(1, 1), (2, 3), (3, 16), (8, 5)])
@pytest.mark.parametrize("boxes", [False, True])
def test_arm_shapes(port, joints, spl, boxes):
    rng = np.random.default_rng(joints)
    dh = W.dh_arm(rng, joints)
    world = W.box_world(rng, 700, free_radius=0.3) if boxes else W.sphere_world(rng, 700, free_radius=0.3)
    for n in (40, 1500):
        s1, s2 = _edges(rng, n, joints, "rv")
        _compare(port, "rv", dh, world, spl, 0.05, s1, s2, boxes=boxes)


def test_worlds(port):
    """Few obstacles, obstacles far off, touching the base, of zero and of large radius."""
    rng = np.random.default_rng(1)
    dh = W.dh_arm(np.random.default_rng(2))
    s1, s2 = _edges(rng, 900, 7, "rv")
    for world in ([[0.9, 0.1, 0.2, 0.1]], [[50.0, 50.0, 50.0, 0.1], [0.5, 0.0, 0.3, 0.0]],
                  [[0.0, 0.0, 0.0, 0.01]], [[0.8, 0.8, 0.8, 0.9], [-1.2, 0.2, 0.4, 0.4]]):
        _compare(port, "rv", dh, np.array(world), 8, 0.05, s1, s2)
        _compare(port, "rv", dh, np.array(world), 8, 0.0, s1[:50], s2[:50])


def test_identical_and_near_pi_edges(port):
    rng = np.random.default_rng(8)
    dh = W.dh_arm(np.random.default_rng(2))
    world = W.sphere_world(rng, 1500)
    s1, s2 = _edges(rng, 1200, 7, "wrap")
    s2[:300] = s1[:300]
    s2[300:600, 3] = s1[300:600, 3] + np.where(s1[300:600, 3] > 0, -PI, PI)  # differences of pi, up to rounding
    s2[600:700] = np.nextafter(s1[600:700], 10.0)
    _compare(port, "wrap", dh, world, 8, 0.05, s1, s2)


def test_without_first_index():
    """The C entry takes null first_j / nd: the same ok for small and large batches."""
    import ctypes as C
    rng = np.random.default_rng(3)
    space = B.RealVectorStateSpace(7, -PI, PI)
    space.setLongestValidSegmentFraction(1.0 / 600)
    ck = B.DHSphereArmValidityChecker(space, W.dh_arm(np.random.default_rng(2)), W.sphere_world(rng, 1500))
    mv = B.DiscreteMotionValidator(ck)
    for n in (5, 700, 5000):
        s1, s2 = _edges(rng, n, 7, "rv")
        a, b = torch.as_tensor(s1, device="cuda"), torch.as_tensor(s2, device="cuda")
        for p in ("fp64", "fp32_guarded"):
            ck.setPrecision(p)
            ok = torch.empty(n, dtype=torch.uint8, device="cuda")
            st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
            capi.check(capi.lib().gbo_check_motion(ck._h, C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr()), n, 7,
                                                   capi.LAYOUT_AOS, capi.SCHEDULE_WARP, C.c_void_p(ok.data_ptr()), None,
                                                   None, st))
            assert torch.equal(ok, mv.checkMotions(a, b)["ok"])


def test_non_finite_edges():
    """Both precisions agree on edges with NaN or infinite coordinates."""
    rng = np.random.default_rng(4)
    space = B.RealVectorStateSpace(7, -PI, PI)
    space.setLongestValidSegmentFraction(1.0 / 600)
    ck = B.DHSphereArmValidityChecker(space, W.dh_arm(np.random.default_rng(2)), W.sphere_world(rng, 1500))
    mv = B.DiscreteMotionValidator(ck)
    s1, s2 = _edges(rng, 40, 7, "rv")
    s1[3, 2] = s2[7, 5] = float("nan")
    out = []
    for p in ("fp64", "fp32_guarded"):
        ck.setPrecision(p)
        out.append(mv.checkMotions(s1, s2))
    for key in ("ok", "first_j", "nd"):
        assert np.array_equal(out[0][key], out[1][key])

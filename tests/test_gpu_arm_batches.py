"""DH arm motion checking around the size of a small batch and the length of a run of states: ok, first invalid index and
segment count of the oracle."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from ompl_gb300 import base as B  # noqa: E402
from ompl_gb300 import capi
from ompl_gb300 import workloads as W  # noqa: E402
from oracle.oracle import CheckerDesc, Oracle, SpaceDesc  # noqa: E402

PI = math.pi
FRACTION = 1.0 / 2500


@pytest.mark.parametrize("n", [300, 4095, 4096, 4097])
def test_run_lengths(n):
    """Edges of 1 to 2,000 states, those next to multiples of a run and of 32 runs among them, some of them repeated
    and of no length."""
    rng = np.random.default_rng(n)
    steps = np.array([1, 2, 31, 32, 33, 63, 64, 65, 1023, 1024, 1025, 1056, 1057, 2000])[rng.integers(0, 14, n)]
    u = rng.normal(size=(n, 7))
    u *= (steps[:, None] - 0.5) * FRACTION * math.sqrt(7) * 2 * PI / np.linalg.norm(u, axis=1, keepdims=True)
    s1 = rng.uniform(-PI, PI, size=(n, 7))
    s2 = s1 + u
    s2[::17] = s1[::17]
    world, dh = W.sphere_world(rng, 1500), W.dh_arm(np.random.default_rng(2))
    space = B.RealVectorStateSpace(7, -PI, PI)
    space.setLongestValidSegmentFraction(FRACTION)
    port = Oracle.port()
    port.set_threads(16)
    sd = SpaceDesc(0, 7, np.full(7, -PI), np.full(7, PI), lvs_fraction=FRACTION)
    ref = port.check_motion(sd, CheckerDesc(W.CHECK_DH_SPHERES, world, dh, 8, 0.05), s1, s2, want_state=False,
                            want_bisect=False)
    assert set(np.unique(ref["nd"])) >= {0, 31, 32, 33, 1024, 1025}
    ck = B.DHSphereArmValidityChecker(space, dh, world)
    mv = B.DiscreteMotionValidator(ck)
    for p in ("fp64", "fp32_guarded"):
        ck.setPrecision(p)
        for a, b in ((s1, s2), (torch.as_tensor(s1, device="cuda"), torch.as_tensor(s2, device="cuda"))):
            r = mv.checkMotions(a, b)
            for key in ("ok", "first_j", "nd"):
                assert np.array_equal(np.asarray(r[key].cpu() if torch.is_tensor(r[key]) else r[key]), ref[key]), (p, key)


@pytest.mark.parametrize("n", [1, 500, 2047, 2048, 2049, 4096])
def test_missing_outputs(n):
    """first_j and nd may each be null: the other outputs are those of a call with both."""
    rng = np.random.default_rng(n)
    space = B.RealVectorStateSpace(7, -PI, PI)
    space.setLongestValidSegmentFraction(1.0 / 600)
    ck = B.DHSphereArmValidityChecker(space, W.dh_arm(np.random.default_rng(2)), W.sphere_world(rng, 1500))
    a = rng.uniform(-PI, PI, size=(n, 7))
    b = np.clip(a + rng.normal(0, 0.3, size=(n, 7)), -PI, PI)
    a, b = torch.as_tensor(a, device="cuda"), torch.as_tensor(b, device="cuda")
    mv = B.DiscreteMotionValidator(ck)
    for p in ("fp64", "fp32_guarded"):
        ck.setPrecision(p)
        want = mv.checkMotions(a, b)
        for with_first, with_nd in ((False, False), (True, False), (False, True)):
            ok = torch.full((n,), 9, dtype=torch.uint8, device="cuda")
            fj, nd = (torch.full((n,), -7, dtype=torch.int32, device="cuda") for _ in range(2))
            ptr = lambda x, there=True: C.c_void_p(x.data_ptr()) if there else None  # noqa: E731
            capi.check(capi.lib().gbo_check_motion(ck._h, ptr(a), ptr(b), n, 7, capi.LAYOUT_AOS, capi.SCHEDULE_WARP,
                                                   ptr(ok), ptr(fj, with_first), ptr(nd, with_nd),
                                                   C.c_void_p(torch.cuda.current_stream().cuda_stream)))
            assert torch.equal(ok, want["ok"])
            assert not with_first or torch.equal(fj, want["first_j"])
            assert not with_nd or torch.equal(nd, want["nd"])

"""The circle checker's cell lists: validity and motion results of the oracle's loop over all circles, for
worlds of one to many circles, of sizes from points to the whole box, far from the origin, and for states
on and around the circles, outside their box and not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from ompl_gb300 import base as B  # noqa: E402
from ompl_gb300 import workloads as W  # noqa: E402
from oracle.oracle import CheckerDesc, Oracle, SpaceDesc  # noqa: E402


def _world(rng, name):
    if name == "one":
        return np.array([[0.4, 0.6, 0.2]])
    if name == "points":
        return np.hstack([rng.uniform(0, 1, (50, 2)), np.zeros((50, 1))])
    if name == "many":
        return W.circles_world(rng, 20_000, 0.0005, 0.003)
    if name == "huge":
        return np.hstack([rng.uniform(0, 1, (3000, 2)), rng.uniform(0.0, 0.6, (3000, 1)) ** 8])
    if name == "negative":
        return np.hstack([rng.uniform(0, 1, (60, 2)), rng.uniform(-0.05, 0.05, (60, 1))])
    if name == "far":
        return np.hstack([rng.uniform(0, 1, (200, 2)) + 1e9, rng.uniform(0.01, 0.05, (200, 1))])
    if name == "infinite":
        return np.array([[0.5, 0.5, 0.1], [np.inf, 0.2, 0.3], [0.1, np.nan, 0.2]])
    return W.circles_world(rng)


@pytest.mark.parametrize("name", ["usual", "one", "points", "many", "huge", "negative", "far", "infinite"])
def test_states_and_edges(name):
    rng = np.random.default_rng(11)
    port = Oracle.port()
    world = _world(rng, name)
    off = 1e9 if name == "far" else 0.0
    low, high = np.full(2, off - 0.5), np.full(2, off + 1.5)
    space = B.RealVectorStateSpace(2, low, high)
    sd = SpaceDesc(0, 2, low, high, lvs_fraction=0.01)
    cd = CheckerDesc(W.CHECK_CIRCLES, world)
    ck = B.CirclesValidityChecker(space, world)
    st = rng.uniform(low, high, size=(20_000, 2))
    # on the circles, up to rounding
    c = world[rng.integers(0, len(world), 4000)]
    t = rng.uniform(0, 2 * np.pi, 4000)
    st[:4000] = c[:, :2] + np.abs(c[:, 2:]) * np.stack([np.cos(t), np.sin(t)], 1)
    st = np.where(np.isfinite(st), st, 0.5)
    assert np.array_equal(ck.isValid(st), port.is_valid(sd, cd, st).astype(bool))
    mv = B.DiscreteMotionValidator(ck)
    for n in (1, 33, 2433, 9999):
        s1, s2 = st[rng.integers(0, len(st), n)], st[rng.integers(0, len(st), n)]
        ref = port.check_motion(sd, cd, s1, s2, want_state=False, want_bisect=False)
        r = mv.checkMotions(s1, s2)
        for key in ("ok", "first_j", "nd"):
            assert np.array_equal(r[key], ref[key]), (n, key)


def test_non_finite_states():
    rng = np.random.default_rng(2)
    ck = B.CirclesValidityChecker(B.RealVectorStateSpace(2, 0.0, 1.0), W.circles_world(rng))
    st = np.array([[np.nan, 0.5], [0.5, np.inf], [-np.inf, 0.1], [1e300, 0.5]])
    assert ck.isValid(st).all()  # no comparison with a NaN or infinite distance holds

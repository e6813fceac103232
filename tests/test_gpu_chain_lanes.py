"""Large kinematic-chain batches (lane per state, world masks): validity and motion results of the FP64 form and
the oracle, over link counts and world sizes on both sides of the masks' limit, with links nearly parallel to world
segments, short and far segments, joint differences at pi and identical end points."""
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

PI = np.pi


def _world(rng, n, name):
    w = W.segment_world(rng, n)
    if name == "short":
        w[:, 2:] = w[:, :2] + rng.normal(0, 1, (n, 2)) * 10.0 ** rng.uniform(-9, -1, (n, 1))
    if name == "sparse":  # most states valid
        w = rng.uniform(0.35, 1.0, (n, 1)) * np.stack([np.cos(t := rng.uniform(0, 2 * PI, n)), np.sin(t)], 1)
        w = np.hstack([w, w + rng.normal(0, 0.05, (n, 2))])
    return np.ascontiguousarray(w)


def _states(rng, world, n, links):
    """Uniform states, a quarter of them with one link's direction within 1e-10 .. 1e-3 of a world segment's."""
    st = rng.uniform(-PI, PI, size=(n, links))
    m = n // 4
    j, k = rng.integers(0, len(world), m), rng.integers(0, links, m)
    phi = np.arctan2(world[j, 3] - world[j, 1], world[j, 2] - world[j, 0])
    phi += rng.choice([-1, 1], m) * 10.0 ** rng.uniform(-10, -3, m) + rng.integers(0, 2, m) * PI
    rows = np.arange(m)
    before = np.where(np.arange(links) < k[:, None], st[:m], 0).sum(1)
    st[rows, k] = (phi - before + PI) % (2 * PI) - PI
    return st


@pytest.mark.parametrize("links,segments,name", [(1, 3, "usual"), (2, 64, "usual"), (6, 64, "short"), (10, 32, "usual"),
                                                 (10, 32, "sparse"), (10, 65, "usual"), (15, 40, "sparse"),
                                                 (10, 1, "usual"), (10, 64, "short"), (7, 20, "sparse")])
def test_states_and_edges(links, segments, name):
    rng = np.random.default_rng(links * 100 + segments)
    world = _world(rng, segments, name)
    space = B.KinematicChainSpace(links, 1.0 / links)
    space.setLongestValidSegmentFraction(0.02)
    ck = B.KinematicChainValidityChecker(space, world)
    n = 131_075
    st = _states(rng, world, n, links)
    a = torch.as_tensor(st, device="cuda")
    want = ck.isValid(a)
    ck.setPrecision("fp32_guarded")
    for count in (32_767, 32_768, n):
        assert torch.equal(ck.isValid(a[:count].contiguous()), want[:count])
        assert torch.equal(ck.isValid(a[:count].T.contiguous(), soa=True), want[:count])
    port = Oracle.port()
    port.set_threads(16)
    sd = SpaceDesc(2, links, link_length=1.0 / links, lvs_fraction=0.02)
    cd = CheckerDesc(W.CHECK_CHAIN_SEGMENTS, world)
    assert np.array_equal(want[:20_000].cpu().numpy().astype(bool), port.is_valid(sd, cd, st[:20_000]).astype(bool))
    # edges from valid states where there are some; some identical, some with a joint difference at pi
    v = st[want.cpu().numpy().astype(bool)]
    s1 = v[rng.integers(0, len(v), n)] if len(v) else st.copy()
    s2 = st[rng.integers(0, n, n)]
    near = rng.random(n) < 0.5
    s2[near] = np.clip(s1[near] + rng.normal(0, 0.05, (near.sum(), links)), -PI, PI)
    s2[:500] = s1[:500]
    s2[500:1000, 0] = s1[500:1000, 0] + np.where(s1[500:1000, 0] > 0, -PI, PI)
    t1, t2 = torch.as_tensor(s1, device="cuda"), torch.as_tensor(s2, device="cuda")
    mv = B.DiscreteMotionValidator(ck)
    for sch in (capi.SCHEDULE_WARP, capi.SCHEDULE_AUTO):
        r = mv.checkMotions(t1, t2, schedule=sch)
        soa = mv.checkMotions(t1.T.contiguous(), t2.T.contiguous(), schedule=sch, soa=True)
        ref = mv.checkMotions(t1, t2, schedule=capi.SCHEDULE_TILE)
        for key in ("ok", "first_j", "nd"):
            assert torch.equal(r[key], ref[key]) and torch.equal(soa[key], ref[key]), (sch, key)
    o = port.check_motion(sd, cd, s1[:20_000], s2[:20_000], want_state=False, want_bisect=False)
    for key in ("ok", "first_j", "nd"):
        assert np.array_equal(r[key][:20_000].cpu().numpy(), o[key]), key


@pytest.mark.parametrize("n", [32_767, 32_768, 100_003])
def test_host_arrays(n):
    """The host calls with page-locked and pageable arrays give the device calls' results."""
    import ctypes as C

    rng = np.random.default_rng(n)
    world = _world(rng, 32, "sparse")
    space = B.KinematicChainSpace(10, 0.1)
    space.setLongestValidSegmentFraction(0.02)
    ck = B.KinematicChainValidityChecker(space, world)
    ck.setPrecision("fp32_guarded")
    a, b = (torch.as_tensor(_states(rng, world, n, 10)) for _ in range(2))
    valid = ck.isValid(a.cuda()).cpu()
    ok = torch.empty(n, dtype=torch.uint8, device="cuda")
    fj, nd = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    da, db = a.cuda(), b.cuda()
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    capi.check(capi.lib().gbo_check_motion(ck._h, ptr(da), ptr(db), n, 10, capi.LAYOUT_AOS, capi.SCHEDULE_AUTO, ptr(ok),
                                           ptr(fj), ptr(nd), None))
    torch.cuda.synchronize()
    for pin in (False, True):
        out = torch.full((2, n), 7, dtype=torch.uint8)
        s1, s2 = a, b
        if pin:
            s1, s2, out = s1.pin_memory(), s2.pin_memory(), out.pin_memory()
        capi.check(capi.lib().gbo_is_valid_host(ck._h, ptr(s1), n, ptr(out[0])))
        capi.check(capi.lib().gbo_check_motion_host(ck._h, ptr(s1), ptr(s2), n, ptr(out[1]), None, None))
        assert torch.equal(out[0], valid) and torch.equal(out[1], ok.cpu())

"""Small host batches (one copy each way on the caller's stream): the results of the device-tensor calls on
both sides of the size limit, ordered after work already queued on the stream, from several threads."""
import threading

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
    pts = torch.as_tensor(rng.uniform(-PI, PI, size=(n, 7)), device="cuda")
    return rng, ck, nn, pts


@pytest.mark.parametrize("n", [0, 1, 3, 291, 292, 293, 584, 586, 1170, 1171])
def test_rows_equal_tensors(n):
    rng, ck, nn, pts = _setup()
    nn.add(pts)
    a, b = rng.uniform(-PI, PI, size=(n, 7)), rng.uniform(-PI, PI, size=(n, 7))
    ta, tb = torch.as_tensor(a, device="cuda"), torch.as_tensor(b, device="cuda")
    assert np.array_equal(ck.isValid(a), ck.isValid(ta).cpu().numpy().astype(bool))
    mv = B.DiscreteMotionValidator(ck)
    r, t = mv.checkMotions(a, b), mv.checkMotions(ta, tb)
    for key in ("ok", "first_j", "nd"):
        assert r[key].dtype == t[key].cpu().numpy().dtype and np.array_equal(r[key], t[key].cpu().numpy())
    assert mv.getValidMotionCount() == int(r["ok"].sum()) and mv.getInvalidMotionCount() == n - int(r["ok"].sum())
    for k in (1, 10):
        (i, d), (ti, td) = nn.nearestK(a, k), nn.nearestK(ta, k)
        assert np.array_equal(i, ti.cpu().numpy()) and np.array_equal(d, td.cpu().numpy())


def test_ordered_after_the_stream():
    rng, _, nn, pts = _setup(200_000)
    q = rng.uniform(-PI, PI, size=(1, 7))
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        x = pts.clone()
        for _ in range(200):  # queued work before the elements are written
            x = x * 1.0
        nn.add(x)
        i, d = nn.nearestK(q, 3)
    ref = torch.linalg.norm(pts - torch.as_tensor(q, device="cuda"), dim=1).topk(3, largest=False)
    assert np.array_equal(i[0], ref.indices.cpu().numpy())


def test_threads():
    rng, ck, nn, pts = _setup()
    nn.add(pts)
    torch.cuda.synchronize()
    mv = B.DiscreteMotionValidator(ck)
    a, b = rng.uniform(-PI, PI, size=(64, 7)), rng.uniform(-PI, PI, size=(64, 7))
    want = [mv.checkMotions(a[i:i + 1], b[i:i + 1])["first_j"][0] for i in range(64)]
    near = [nn.nearestK(a[i:i + 1], 1)[0][0, 0] for i in range(64)]
    got, bad = {}, []

    def work(t):
        try:
            for i in range(t, 64, 4):
                got[i] = (mv.checkMotions(a[i:i + 1], b[i:i + 1])["first_j"][0])
        except Exception as e:  # reported below
            bad.append(e)

    ts = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad and [got[i] for i in range(64)] == want
    assert near == [nn.nearestK(a[i:i + 1], 1)[0][0, 0] for i in range(64)]

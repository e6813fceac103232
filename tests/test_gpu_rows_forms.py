"""Host-array arguments: what numpy batches are refused whatever their size, and calls from several threads."""
import threading
import time

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


@pytest.mark.parametrize("rows", [2, 3000])  # below and above the size of a small batch
def test_refused(rows):
    _, ck, nn = _setup()
    text = [["0.1"] * 7] * rows
    with pytest.raises(TypeError):
        ck.isValid(text)
    with pytest.raises(TypeError):
        B.DiscreteMotionValidator(ck).checkMotions(text, text)
    with pytest.raises(TypeError):
        nn.nearestK(text, 1)
    with pytest.raises(TypeError):
        nn.nearestK(np.zeros((rows, 7)), 2.5)
    for k in (-1, 0, 65):
        with pytest.raises((RuntimeError, ValueError)):
            nn.nearestK(np.zeros((rows, 7)), k)
    # converted as before
    a = np.zeros((rows, 7), dtype=np.float32)
    assert np.array_equal(ck.isValid(a), ck.isValid(a.astype(np.float64)))
    assert np.array_equal(nn.nearestK(a.astype(np.int32).tolist(), np.int64(3))[0], nn.nearestK(a, 3)[0])


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


def test_all_calls_from_threads():
    """isValid, checkMotions and nearestK from four threads at once, with batches whose sizes differ (the buffers grow
    meanwhile): the results of the same calls made one after another."""
    rng, ck, nn = _setup()
    mv = B.DiscreteMotionValidator(ck)
    sizes = [1, 3, 17, 64, 120, 290]
    batches = [(rng.uniform(-PI, PI, size=(n, 7)), rng.uniform(-PI, PI, size=(n, 7)), 1 + n % 9) for n in sizes * 8]

    def calls(b):
        a, c, k = b
        m = mv.checkMotions(a, c)
        i, d = nn.nearestK(a, k)
        return [ck.isValid(a), m["ok"], m["first_j"], m["nd"], i, d]

    want = [calls(b) for b in batches]
    rng, ck, nn = _setup()  # buffers of no size yet
    mv = B.DiscreteMotionValidator(ck)
    got, bad = {}, []

    def work(t):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for i in range(t, len(batches), 4):
                    got[i] = calls(batches[i])
        except Exception as e:  # reported below
            bad.append(e)

    ts = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
    for i, w in enumerate(want):
        assert all(np.array_equal(x, y) for x, y in zip(got[i], w)), i


def test_a_waiting_thread_holds_up_no_other():
    """A thread whose stream has queued work waits for it in its call; another thread's call on another stream does
    not."""
    rng, ck, _ = _setup()
    mv = B.DiscreteMotionValidator(ck)
    a = rng.uniform(-PI, PI, size=(4, 7))
    for _ in range(3):
        ck.isValid(a), mv.checkMotions(a, a)
    slow, quick = torch.cuda.Stream(), torch.cuda.Stream()
    done = []

    def held():
        with torch.cuda.stream(slow):
            torch.cuda._sleep(1_500_000_000)  # most of a second of clock cycles
            ck.isValid(a)
            done.append(time.perf_counter())

    t = threading.Thread(target=held)
    t.start()
    time.sleep(0.1)
    with torch.cuda.stream(quick):
        ck.isValid(a)
        mv.checkMotions(a, a)
    free = time.perf_counter()
    t.join()
    assert done[0] > free


def test_large_lists_are_converted_once():
    """A batch too large for the row buffers goes on as the array that its size was taken from."""
    rng, ck, nn = _setup()
    made = []

    class Counted:
        def __init__(self, a):
            self.a = a

        def __array__(self, dtype=None, copy=None):
            made.append(1)
            return self.a if dtype is None else self.a.astype(dtype)

    a, b = rng.uniform(-PI, PI, size=(3000, 7)), rng.uniform(-PI, PI, size=(3000, 7))
    assert np.array_equal(ck.isValid(Counted(a)), ck.isValid(a)) and len(made) == 1
    mv = B.DiscreteMotionValidator(ck)
    assert np.array_equal(mv.checkMotions(Counted(a), Counted(b))["first_j"], mv.checkMotions(a, b)["first_j"])
    assert len(made) == 3
    assert np.array_equal(nn.nearestK(Counted(a), 3)[0], nn.nearestK(a, 3)[0]) and len(made) == 4


def test_a_host_batch_in_a_capture():
    """It is refused, since it waits for its results, and leaves no error for the calls after it."""
    rng, ck, nn = _setup()
    a = rng.uniform(-PI, PI, size=(4, 7))
    want, near = ck.isValid(a), nn.nearestK(a, 3)[0]
    for call in (lambda: ck.isValid(a), lambda: nn.nearestK(a, 3)):
        torch.cuda.synchronize()
        with pytest.raises(RuntimeError):
            with torch.cuda.graph(torch.cuda.CUDAGraph()):
                call()
        assert np.array_equal(ck.isValid(a), want)
        assert np.array_equal(nn.nearestK(a, 3)[0], near)

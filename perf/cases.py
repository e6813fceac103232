"""Performance cases of the sampling / validity / motion / nearest-neighbour path: what a planner or a
roadmap builder asks of this package through its Python classes, from one query and one edge of a
growing tree to a whole two-million-sample roadmap.

A case is a dict of plain values; `prepare` makes what the program has in hand (worlds, indexes,
samplers, batches of states), `run` makes one pass, `work` says what the pass cannot do without and
`exact` gives the floating outputs in 64 bits without this package's code.

Worlds, states and edges follow `ompl_gb300.workloads`, drawn on the GPU from the seed; the DH arm is
the one of the repository's arm workloads (its seven rows are part of the robot, not of the input).
"""
import math

import numpy as np
import torch

from ompl_gb300 import base as B
from ompl_gb300 import capi, prm
from ompl_gb300 import workloads as W

PI = math.pi
DEV = "cuda"

# What each listed size stands for:
#   tree_extend          one extension of an RRT tree, the drop-in calls of a single planner: the nearest
#                        of 2,000 motions to a sample and one checkMotion towards it. Latency counts.
#   circles_10k          the plain 2-D configuration at its own size: validity of 10,000 states, 10,000
#                        edges, k = 10 neighbours of 1,000 queries; small, FP64.
#   chain_states_1m      validity filter of a million samples of the 10-link chain.
#   chain_edges_100k     lazy-PRM style re-check of 100,000 chain edges between valid states.
#   chain_knn_20k        k = 16 neighbours of 20,000 states in a million-state chain index.
#   arm_edges_256k       256,000 arm edges of 2..2,000 steps, the largest edge batch.
#   arm_box_edges_3k     an ordinary batch of edges among boxes in the default precision and schedule, as
#                        a program gets them without setting either; odd size.
#   roadmap_knn_500      one planner's query batch against its own 60,000-state roadmap.
#   radius_1k            RRT* / PRM* rewiring sets: all neighbours within a radius, 1,000 queries.
#   uniform_1m           a million uniform samples from one stream.
#   gaussian_100k        100,003 Gaussian samples around given means (bridge / Gaussian samplers).
#   prm_2m               a whole PRM roadmap: samples, filter, prefix neighbours, edges.


def listed():
    return [
        {"name": "tree_extend", "op": "extend", "tree": 2000, "spheres": 4096},
        {"name": "circles_10k", "op": "circles", "states": 10000, "edges": 10000, "queries": 1000, "k": 10},
        {"name": "chain_states_1m", "op": "chain_states", "links": 10, "n": 1000000},
        {"name": "chain_edges_100k", "op": "chain_edges", "links": 10, "n": 100000},
        {"name": "chain_knn_20k", "op": "knn", "space": "chain", "dim": 10, "index": 1000000, "queries": 20000,
         "k": 16},
        {"name": "arm_edges_256k", "op": "arm_edges", "n": 256000, "obstacles": "spheres", "world": 4096,
         "batched": True},
        {"name": "arm_box_edges_3k", "op": "arm_edges", "n": 3001, "obstacles": "boxes", "world": 2048,
         "batched": False},
        {"name": "roadmap_knn_500", "op": "knn", "space": "wrap", "dim": 7, "index": 60000, "queries": 500, "k": 10},
        {"name": "radius_1k", "op": "radius", "dim": 7, "index": 50000, "queries": 1000, "target": 30},
        {"name": "uniform_1m", "op": "uniform", "dim": 10, "n": 1000000},
        {"name": "gaussian_100k", "op": "gaussian", "dim": 7, "n": 100003},
        {"name": "prm_2m", "op": "prm", "samples": 2000000, "spheres": 16384, "k": 10},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["extend", "circles", "chain_states", "chain_edges", "knn", "knn", "arm_edges", "arm_edges",
                     "radius", "uniform", "gaussian", "prm"])
    if op == "extend":
        return {"op": op, "tree": log(100, 20000), "spheres": log(1024, 8192)}
    if op == "circles":
        return {"op": op, "states": log(1000, 50000), "edges": log(1000, 50000), "queries": log(10, 5000),
                "k": rng.randint(1, 16)}
    if op == "chain_states":
        return {"op": op, "links": rng.randint(6, 12), "n": log(20000, 1000000)}
    if op == "chain_edges":
        return {"op": op, "links": rng.randint(8, 12), "n": log(16, 100000)}
    if op == "knn":
        space = rng.choice(["chain", "wrap", "wrap", "rv"])
        # the serving range (10k..200k states, 1..4,096 queries), and the large chain index's
        big = space == "chain" and rng.random() < 0.5
        return {"op": op, "space": space, "dim": rng.randint(6, 10) if space == "chain" else rng.randint(3, 8),
                "index": log(200000, 1000000) if big else log(10000, 200000),
                "queries": log(1000, 20000) if big else log(1, 4096), "k": rng.randint(1, 16)}
    if op == "arm_edges":
        batched = rng.random() < 0.7
        return {"op": op, "n": log(16, 256000) if batched else log(16, 8192),
                "obstacles": rng.choice(["spheres", "spheres", "boxes"]), "world": log(1024, 16384),
                "batched": batched}
    if op == "radius":
        return {"op": op, "dim": rng.randint(2, 8), "index": log(1000, 100000), "queries": log(1, 2000),
                "target": rng.randint(5, 100)}
    if op in ("uniform", "gaussian"):
        return {"op": op, "dim": rng.randint(2, 12), "n": log(100, 1000000 if op == "uniform" else 500000)}
    return {"op": op, "samples": log(20000, 1000000), "spheres": log(1024, 16384), "k": rng.randint(5, 15)}


# ---------------------------------------------------------------- inputs
def _gen(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFF)
    return g


def _uniform(g, n, dim, lo, hi):
    return torch.rand((n, dim), generator=g, device=DEV, dtype=torch.float64) * (hi - lo) + lo


def _arm_space(wrap=False):
    low, high = np.full(7, -PI), np.full(7, PI)
    if wrap:  # the roadmap's joint space, edges at 0.01 rad
        s = B.WrapL2StateSpace(7)
        s.setLongestValidSegmentFraction(0.01 / math.sqrt(7 * PI * PI))
    else:
        s = B.RealVectorStateSpace(7, low, high)
        s.setLongestValidSegmentFraction(1.0 / 2500.0)
    return s


def _arm_checker(space, rng, n, obstacles="spheres"):
    dh = W.dh_arm(np.random.default_rng(2))
    if obstacles == "boxes":
        return B.DHBoxArmValidityChecker(space, dh, W.box_world(rng, n))
    return B.DHSphereArmValidityChecker(space, dh, W.sphere_world(rng, n))


def _arm_edges(seed, n, lvs):
    """Edges of log-uniform 2..2,000 steps inside the joint box (workloads.arm_edges on the GPU)."""
    g = _gen(seed, 5)
    steps = torch.floor(torch.exp(_uniform(g, n, 1, math.log(2.0), math.log(2000.0))))
    length = (steps - 0.5) * lvs
    s1 = torch.empty((n, 7), device=DEV, dtype=torch.float64)
    s2 = torch.empty_like(s1)
    todo = torch.arange(n, device=DEV)
    while todo.numel():
        u = torch.randn((todo.numel(), 7), generator=g, device=DEV, dtype=torch.float64)
        step = u / torch.linalg.norm(u, dim=1, keepdim=True) * length[todo]
        fit = (step.abs() < 2 * PI).all(1)
        i, st = todo[fit], step[fit]
        lo, hi = -PI - torch.clamp(st, max=0.0), PI - torch.clamp(st, min=0.0)
        a = lo + (hi - lo) * torch.rand(st.shape, generator=g, device=DEV, dtype=torch.float64)
        s1[i], s2[i] = a, torch.clamp(a + st, -PI, PI)
        todo = todo[~fit]
    return s1, s2


def _chain(seed, links):
    space = B.KinematicChainSpace(links, 1.0 / links)
    space.setLongestValidSegmentFraction(0.005)
    rng = np.random.default_rng([int(seed), 11])
    checker = B.KinematicChainValidityChecker(space, W.segment_world(rng))
    checker.setPrecision("fp32_guarded")
    return space, checker


def _index_points(case, seed):
    return _uniform(_gen(seed, 21), case["index"], case["dim"], -PI, PI)


def _knn_space(case):
    if case["space"] == "chain":
        return B.KinematicChainSpace(case["dim"], 0.1)
    if case["space"] == "wrap":
        return B.WrapL2StateSpace(case["dim"])
    return B.RealVectorStateSpace(case["dim"], -PI, PI)


def _queries(case, seed):
    return _uniform(_gen(seed, 22), case["queries"], case["dim"], -PI, PI)


def _radius(case):
    """A radius that holds about `target` of the uniform index's elements (away from the bounds)."""
    d = case["dim"]
    ball = PI ** (d / 2) / math.gamma(d / 2 + 1)
    return 2 * PI * (case["target"] / (case["index"] * ball)) ** (1.0 / d)


def _room(case):
    """How many neighbours the padded outputs of a radius search hold (the count varies with the inputs)."""
    return 2 * case["target"] * case["queries"] + 1024


def _stream_seed(seed):
    return (int(seed) * 2654435761 + 97) & 0xFFFFFFFF


def prepare(case, seed):
    op = case["op"]
    s = {"op": op}
    if op == "extend":
        space = _arm_space()
        checker = _arm_checker(space, np.random.default_rng([int(seed), 1]), case["spheres"])
        # the tree's motions are valid states
        pool = _uniform(_gen(seed, 3), 16 * case["tree"] + 4096, 7, -PI, PI)
        checker.setPrecision("fp32_guarded")
        tree = pool[checker.isValid(pool).bool()][:case["tree"]].contiguous()
        checker.setPrecision("fp64")
        nn = B.NearestNeighborsGPU(space, capacity=2 * case["tree"])
        nn.add(tree)
        q = np.random.default_rng([int(seed), 4]).uniform(-PI, PI, size=(1, 7))
        s.update(nn=nn, tree=tree.cpu().numpy(), q=q, mv=B.DiscreteMotionValidator(checker),
                 range=0.2 * space.getMaximumExtent())
    elif op == "circles":
        rng = np.random.default_rng([int(seed), 2])
        space = B.RealVectorStateSpace(2, 0.0, 1.0)
        checker = B.CirclesValidityChecker(space, W.circles_world(rng))
        g = _gen(seed, 6)
        states = _uniform(g, case["states"], 2, 0.0, 1.0)
        i = torch.randint(case["states"], (case["edges"],), generator=g, device=DEV)
        j = torch.randint(case["states"], (case["edges"],), generator=g, device=DEV)
        nn = B.NearestNeighborsGPU(space, capacity=case["states"])
        nn.add(states)
        s.update(checker=checker, mv=B.DiscreteMotionValidator(checker), states=states, s1=states[i].contiguous(),
                 s2=states[j].contiguous(), nn=nn, q=_uniform(g, case["queries"], 2, 0.0, 1.0), k=case["k"])
    elif op == "chain_states":
        _, checker = _chain(seed, case["links"])
        x = _uniform(_gen(seed, 7), case["n"], case["links"], -PI, PI)
        s.update(checker=checker, states=x.T.contiguous())
    elif op == "chain_edges":
        _, checker = _chain(seed, case["links"])
        g, found, have = _gen(seed, 8), [], 0
        for _ in range(16):  # both ends of an edge are valid states, a few in a thousand of the samples
            x = _uniform(g, 1 << 20, case["links"], -PI, PI)
            found.append(x[checker.isValid(x).bool()])
            have += found[-1].shape[0]
            if have >= 4000:
                break
        v = torch.cat(found)
        if v.shape[0] < 2:
            v = x[:2]
        i = torch.randint(v.shape[0], (case["n"],), generator=g, device=DEV)
        j = torch.randint(v.shape[0], (case["n"],), generator=g, device=DEV)
        s.update(mv=B.DiscreteMotionValidator(checker), s1=v[i].T.contiguous(), s2=v[j].T.contiguous(), soa=True,
                 schedule=capi.SCHEDULE_AUTO)
    elif op == "arm_edges":
        space = _arm_space()
        checker = _arm_checker(space, np.random.default_rng([int(seed), 1]), case["world"], case["obstacles"])
        s1, s2 = _arm_edges(seed, case["n"], space.getLongestValidSegmentLength())
        if case["batched"]:
            checker.setPrecision("fp32_guarded")
            s1, s2 = s1.T.contiguous(), s2.T.contiguous()
        s.update(mv=B.DiscreteMotionValidator(checker), s1=s1, s2=s2, soa=case["batched"],
                 schedule=capi.SCHEDULE_AUTO if case["batched"] else capi.SCHEDULE_PLAIN)
    elif op in ("knn", "radius"):
        space = _knn_space(case) if op == "knn" else B.RealVectorStateSpace(case["dim"], -PI, PI)
        nn = B.NearestNeighborsGPU(space, capacity=case["index"])
        nn.add(_index_points(case, seed))
        s.update(nn=nn, q=_queries(case, seed))
        if op == "knn":
            s["k"] = case["k"]
        else:
            s.update(radius=_radius(case), room=_room(case))
    elif op in ("uniform", "gaussian"):
        space = B.RealVectorStateSpace(case["dim"], -PI, PI)
        s.update(sampler=B.StateSampler(space, _stream_seed(seed)), n=case["n"])
        if op == "gaussian":
            s["mean"] = _uniform(_gen(seed, 9), case["n"], case["dim"], -PI, PI)
    else:
        space = _arm_space(wrap=True)
        checker = _arm_checker(space, np.random.default_rng([int(seed), 1]), case["spheres"])
        checker.setPrecision("fp32_guarded")
        s.update(space=space, checker=checker, samples=case["samples"], k=case["k"], seed=_stream_seed(seed))
    torch.cuda.synchronize()
    return s


STDDEV = 0.3


def run(s):
    op = s["op"]
    if op == "extend":
        idx, dist = s["nn"].nearestK(s["q"], 1)
        near = s["tree"][idx[0, 0]]
        d = float(dist[0, 0])
        new = s["q"][0] if d <= s["range"] else near + (s["q"][0] - near) * (s["range"] / d)
        return {"key": idx, "distance": dist, "ok": s["mv"].checkMotion(near, new)}
    if op == "circles":
        m = s["mv"].checkMotions(s["s1"], s["s2"])
        idx, dist = s["nn"].nearestK(s["q"], s["k"])
        return {"valid": s["checker"].isValid(s["states"]), "ok": m["ok"], "first_j": m["first_j"], "nd": m["nd"],
                "key": idx, "distance": dist}
    if op == "chain_states":
        return {"valid": s["checker"].isValid(s["states"], soa=True)}
    if op in ("chain_edges", "arm_edges"):
        m = s["mv"].checkMotions(s["s1"], s["s2"], schedule=s["schedule"], soa=s["soa"])
        return {"ok": m["ok"], "first_j": m["first_j"], "nd": m["nd"]}
    if op == "knn":
        idx, dist = s["nn"].nearestK(s["q"], s["k"])
        return {"key": idx, "distance": dist}
    if op == "radius":
        counts, idx, dist = s["nn"].nearestR(s["q"], s["radius"])
        room = s["room"] - idx.shape[0]
        return {"count": counts, "key": np.pad(idx, (0, room), constant_values=-1),
                "distance": np.pad(dist, (0, room), constant_values=np.inf)}
    if op == "uniform":
        return {"states": s["sampler"].sampleUniform(s["n"], soa=True, host=False)}
    if op == "gaussian":
        return {"states": s["sampler"].sampleGaussian(s["mean"], STDDEV)}
    r = prm.construct_roadmap(s["space"], s["checker"], s["seed"], s["samples"], k=s["k"])
    # the numbers of milestones and edges vary with the world: padded to one shape
    pad = torch.nn.functional.pad
    n, e = s["samples"] - r.sample_index.shape[0], s["samples"] * s["k"] - r.edge_src.shape[0]
    return {"sample_index": pad(r.sample_index, (0, n), value=-1), "milestones": pad(r.milestones, (0, n)),
            "edge_src": pad(r.edge_src, (0, e), value=-1), "edge_dst": pad(r.edge_dst, (0, e), value=-1),
            "candidates": r.candidate_edges, "checked": r.checked_states}


# ---------------------------------------------------------------- work
# Floating-point operations of one state's test, as the repository's benchmark counts them: the chain's
# forward kinematics and its segment pairs; the arm's seven joint transforms and 56 sphere centres with
# about one listed obstacle each. States per edge are those that the ordered check evaluates on these
# workloads (2.4 on the chain, 49 on the arm's 2..2,000-step edges).
def _chain_flops(links):
    return 5 * links + ((links + 1) * links // 2 + (links + 1) * 32) * 21


ARM_FLOPS = 7 * 75 + 56 * 20


def work(case):
    op = case["op"]
    if op == "extend":
        return {"bytes": case["tree"] * 28 + 3 * 56 + 24, "flops": case["tree"] * 21 + 49 * ARM_FLOPS}
    if op == "circles":
        n, m, q, k = case["states"], case["edges"], case["queries"], case["k"]
        return {"bytes": n * 33 + m * 41 + q * (16 + 16 * k), "flops": (n + 20 * m) * 100 * 5 + q * k * 5}
    if op == "chain_states":
        # an invalid state (all but a few in a thousand) takes its kinematics and one intersecting pair
        return {"bytes": case["n"] * (8 * case["links"] + 1), "flops": case["n"] * (5 * case["links"] + 21)}
    if op == "chain_edges":
        return {"bytes": case["n"] * (16 * case["links"] + 9), "flops": 2.4 * case["n"] * _chain_flops(case["links"])}
    if op == "arm_edges":
        return {"bytes": case["n"] * (112 + 9), "flops": 49 * case["n"] * ARM_FLOPS}
    if op in ("knn", "radius"):
        found = case["queries"] * (case["k"] if op == "knn" else case["target"])
        return {"bytes": (case["index"] + case["queries"]) * 8 * case["dim"] + 16 * found,
                "flops": found * 3 * case["dim"]}
    if op in ("uniform", "gaussian"):
        v = case["n"] * case["dim"]
        return {"bytes": v * (8 if op == "uniform" else 16), "flops": v * (2 if op == "uniform" else 20)}
    n, k = case["samples"], case["k"]
    # about 0.31 of the samples are milestones, each with k edges of which two states are checked
    m = 0.31 * n
    return {"bytes": m * (56 + 8 + 16 * k), "flops": n * ARM_FLOPS + 2 * m * k * ARM_FLOPS}


# ---------------------------------------------------------------- the outputs in 64 bits
def _features(x, link):
    t = torch.cumsum(x, 1)
    return torch.cumsum(torch.cos(t), 1) * link, torch.cumsum(torch.sin(t), 1) * link


def _distance(kind, a, b):
    """(rows of a) x (rows of b), or row by row where b has three dimensions (rows, candidates, dim)."""
    b = b if b.dim() == 3 else b[None]
    s = torch.zeros((a.shape[0], b.shape[1]), device=a.device, dtype=a.dtype)
    for d in range(a.shape[1]):
        x = (a[:, None, d] - b[:, :, d]).abs()
        if kind == "wrap":
            x = torch.minimum(x, 2 * PI - x)
        s += x * x
    return s.sqrt()


def _chain_distance(fa, fb):
    xa, ya = fa
    xb, yb = (t if t.dim() == 3 else t[None] for t in fb)
    s = torch.zeros((xa.shape[0], xb.shape[1]), device=xa.device, dtype=xa.dtype)
    for d in range(xa.shape[1]):
        s += ((xa[:, None, d] - xb[:, :, d]) ** 2 + (ya[:, None, d] - yb[:, :, d]) ** 2).sqrt()
    return s


def _nearest(kind, points, q, k, link=0.1):
    """The k smallest distances of each query, ascending: candidates by 32-bit distances with room to
    spare, their distances in 64 bits."""
    keep = min(points.shape[0], k + 64)
    rows = max(1, (1 << 28) // points.shape[0])
    out = []
    if kind == "chain":
        fp = _features(points, link)
        f32 = tuple(t.float() for t in fp)
    for at in range(0, q.shape[0], rows):
        x = q[at:at + rows]
        if kind == "chain":
            fx = _features(x, link)
            c = _chain_distance(tuple(t.float() for t in fx), f32).topk(keep, 1, largest=False).indices
            d = _chain_distance(fx, (fp[0][c], fp[1][c]))
        else:
            c = _distance(kind, x.float(), points.float()).topk(keep, 1, largest=False).indices
            d = _distance(kind, x, points[c])
        d = d.sort(1).values[:, :k]
        if d.shape[1] < k:
            d = torch.nn.functional.pad(d, (0, k - d.shape[1]), value=math.inf)
        out.append(d)
    return torch.cat(out)


def _canonical(seed, count):
    """generate_canonical<double, 53> of a 32-bit Mersenne Twister: `count` values in [0, 1)."""
    bits = np.random.MT19937()
    bits._legacy_seeding(seed)
    w = bits.random_raw(2 * count).astype(np.uint32).astype(np.float64)
    u = (w[0::2] + w[1::2] * 4294967296.0) * 2.0 ** -64
    return np.where(u >= 1.0, np.nextafter(1.0, 0.0), u)


def exact(case, seed):
    op = case["op"]
    if op == "extend":
        # only the distance is a computed number; the tree is the prepared one
        s = prepare(case, seed)
        t = torch.as_tensor(s["tree"], device=DEV)
        d = _nearest("rv", t, torch.as_tensor(s["q"], device=DEV), 1)
        return {"key": None, "distance": d.cpu().numpy(), "ok": None}
    if op == "circles":
        s = prepare(case, seed)
        return {"valid": None, "ok": None, "first_j": None, "nd": None, "key": None,
                "distance": _nearest("rv", s["states"], s["q"], s["k"])}
    if op == "knn":
        return {"key": None, "distance": _nearest(case["space"], _index_points(case, seed), _queries(case, seed),
                                                  case["k"])}
    if op == "radius":
        p, q, r, out = _index_points(case, seed), _queries(case, seed), _radius(case), []
        for at in range(0, q.shape[0], 500):
            d = _distance("rv", q[at:at + 500], p)
            out += [row[row <= r].sort().values for row in d]
        d = torch.cat(out).cpu().numpy()
        return {"count": None, "key": None,
                "distance": np.pad(d, (0, _room(case) - d.shape[0]), constant_values=np.inf)}
    if op == "uniform":
        u = _canonical(_stream_seed(seed), case["n"] * case["dim"]).reshape(case["n"], case["dim"])
        return {"states": np.ascontiguousarray((u * (PI - -PI) + -PI).T)}
    if op == "gaussian":
        m = case["n"] * case["dim"]
        pairs = (m + 1) // 2
        cand = int(pairs / 0.7853981633974483 + 8 * math.sqrt(pairs / 0.7853981633974483) + 64)
        u = _canonical(_stream_seed(seed), 2 * cand).reshape(cand, 2)
        x, y = 2.0 * u[:, 0] - 1.0, 2.0 * u[:, 1] - 1.0
        r2 = x * x + y * y
        at = np.flatnonzero((r2 <= 1.0) & (r2 != 0.0))[:pairs]
        f = np.sqrt(-2.0 * np.log(r2[at]) / r2[at])
        z = np.stack([y[at] * f, x[at] * f], 1).reshape(-1)[:m].reshape(case["n"], case["dim"])
        mean = _uniform(_gen(seed, 9), case["n"], case["dim"], -PI, PI).cpu().numpy()
        return {"states": np.clip(z * STDDEV + mean, -PI, PI)}
    return None

"""Timed cases of the framework: what programs have it do, through its public entry points.

The sizes and radii come from the benchmark's workloads (``ridgedetection_b200/generators.py``:
the 20,000-point sine, the 1M-point helix, the 10M-point tiled spiral, the batch of clouds of 1,000
to 200,000 points, the 262,144-point adjoint) and from the tests; ``draw`` spreads over the ranges
that they span.  All clouds are float32 (the only type the framework takes), in 2 and 3 dimensions.

Kinds of case:
  solve     one cloud, choose -> (evolve -> decimate)* to convergence (BruteForceRidgeDetection)
  tiled     the same over a tile tree (TiledRidgeDetection)
  batch     many clouds in one run (BatchedRidgeDetection)
  choose    the greedy r1-separated subset (rd_choose)
  evolve    one evolve pass from a chosen set (rd_evolve_pass)
  decimate  one decimation of a chosen set (rd_decimate)
  adjoint   a fixed number of evolve passes and their gradient (evolve_function, forward + backward)
  report    what is read off a finished ridge: its chains, and its distance to the ideal curve
"""
import ctypes
import math

import numpy as np
import torch

import ridgedetection_b200 as rdb
from ridgedetection_b200 import _lib as L
from ridgedetection_b200.autograd import evolve_function

# rows of the arrays that a program keeps for a ridge and for a chosen set; what a call does not
# fill stays zero, so that outputs have one shape whatever the number of points found
RIDGE_ROWS = 1_024
CHOSEN_ROWS = 8_192


def listed():
    return [
        # the smallest cloud of the batch, solved alone: latency of a whole solve
        dict(name="solve_sine2d_1k", kind="solve", gen="sine", n=1_000, r1=0.3, r2=0.6,
             layout="row", host=False),
        # the benchmark's first workload, from and to host arrays
        dict(name="solve_sine2d_20k", kind="solve", gen="sine", n=20_000, r1=0.3, r2=0.6,
             layout="row", host=True),
        # an odd mid-size cloud, column-major points on the device
        dict(name="solve_helix3d_77777_col", kind="solve", gen="helix", n=77_777, r1=0.2, r2=0.4,
             layout="col", host=False),
        # the headline workload
        dict(name="solve_helix3d_1m", kind="solve", gen="helix", n=1_000_000, r1=0.15, r2=0.3,
             layout="row", host=False),
        # a tile tree whose dense tiles are subdivided, as in the full-size tests
        dict(name="tiled_spiral2d_1m_split", kind="tiled", n=1_000_000, r1=0.2, r2=0.4,
             tiles=8, capacity=50_000),
        # the benchmark's tiled workload
        dict(name="tiled_spiral2d_10m", kind="tiled", n=10_000_000, r1=0.2, r2=0.4,
             tiles=64, capacity=10_000_001),
        # half the benchmark's batch: the largest call
        dict(name="batch_2048", kind="batch", clouds=2_048, sizes=1, n_min=1_000, n_max=200_000),
        # the device-level steps on the headline cloud, as a host of the pipeline calls them
        dict(name="choose_helix3d_1m", kind="choose", gen="helix", n=1_000_000, r1=0.15),
        dict(name="evolve_helix3d_1m", kind="evolve", gen="helix", n=1_000_000, r1=0.15),
        # the merged chosen set of a tiled run
        dict(name="decimate_spiral2d_10k", kind="decimate", n=10_000, r2=0.075),
        # the adjoint workload: 20 passes, a checkpoint every 5
        dict(name="adjoint_helix3d_262k", kind="adjoint", n=262_144, r1=0.15, iters=20, every=5),
        # chains and quality of a ridge of the size the workloads end with
        dict(name="report_helix3d", kind="report", n=300, ideal=100_000, r2=0.3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "tiled", "tiled", "batch", "choose", "evolve",
                       "evolve", "decimate", "adjoint", "report"])
    gen = rng.choice(["sine", "helix"])
    r1 = round(rng.uniform(0.1, 0.3), 3)
    if kind == "solve":
        return dict(kind=kind, gen=gen, n=_log(rng, 1_000, 1_000_000), r1=r1, r2=round(2 * r1, 3),
                    layout=rng.choice(["row", "row", "col"]), host=rng.random() < 0.3)
    if kind == "tiled":
        n = _log(rng, 100_000, 10_000_000)
        r1 = round(rng.uniform(0.15, 0.25), 3)
        return dict(kind=kind, n=n, r1=r1, r2=round(2 * r1, 3),
                    tiles=rng.randint(24, 64) if n > 2_000_000 else rng.randint(8, 32),
                    capacity=rng.choice([n + 1, 50_000]))
    if kind == "batch":
        return dict(kind=kind, clouds=_log(rng, 16, 1_024), sizes=rng.randint(2, 1_000_000),
                    n_min=1_000, n_max=_log(rng, 10_000, 200_000))
    if kind in ("choose", "evolve"):
        return dict(kind=kind, gen=gen, n=_log(rng, 1_000, 1_000_000), r1=r1)
    if kind == "decimate":
        n = _log(rng, 100, 10_000)
        # about ten neighbours within r2, as a set separated by r1 = r2/2 has
        return dict(kind=kind, n=n, r2=round(0.075 * math.sqrt(10_000 / n), 4))
    if kind == "adjoint":
        return dict(kind=kind, n=_log(rng, 4_000, 262_144), r1=r1, iters=rng.randint(5, 20),
                    every=rng.choice([0, 5]))
    return dict(kind=kind, n=_log(rng, 30, 500), ideal=_log(rng, 10_000, 100_000), r2=0.3)


# --- inputs ---------------------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, n, lo, hi):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _normal(g, shape, sigma):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float64) * sigma


def _sine(g, n):
    t = _uniform(g, n, 0.0, 10.0)
    return torch.stack([t, torch.sin(2.0 * t)], 1) + _normal(g, (n, 2), 0.1)


def _helix(g, n):
    t = _uniform(g, n, 0.0, 8.0 * math.pi)
    return torch.stack([torch.cos(t), torch.sin(t), 0.15 * t], 1) + _normal(g, (n, 3), 0.05)


def _spiral(g, n, clutter):
    """The Archimedean spiral with noise, `clutter` of the points uniform in its bounding box."""
    n_clut = int(round(n * clutter))
    th = _uniform(g, n - n_clut, 0.0, 6.0 * math.pi)
    p = torch.stack([0.5 * th * torch.cos(th), 0.5 * th * torch.sin(th)], 1)
    p += _normal(g, p.shape, 0.05)
    if n_clut:
        lo, hi = p.amin(0), p.amax(0)
        box = torch.rand((n_clut, 2), generator=g, device="cuda", dtype=torch.float64)
        p = torch.cat([p, lo + box * (hi - lo)])
        p = p[torch.randperm(n, generator=g, device="cuda")]
    return p


def _cloud(case, seed):
    g = _generator(seed)
    p = _sine(g, case["n"]) if case["gen"] == "sine" else _helix(g, case["n"])
    return p.float().contiguous()


def _greedy(P, r1):
    """The chosen set of the cloud, in plain torch: each point further than r1 from all chosen so far."""
    left, got = P, []
    r1 = torch.tensor(r1, dtype=torch.float32).item()
    while left.shape[0]:
        got.append(left[0])
        d = left - left[0]
        left = left[(d * d).sum(1) > r1 * r1]
    return torch.stack(got)


def _batch_descs(case):
    """(offset, n, dim, r1, r2) of each cloud, sizes log-uniform, sine and helix in turn."""
    r = np.random.default_rng(case["sizes"])
    descs, off = [], 0
    for c in range(case["clouds"]):
        n = int(round(math.exp(r.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
        r1 = float(np.float32(r.uniform(0.1, 0.3)))
        dim = 2 if c % 2 == 0 else 3
        descs.append((off, n, dim, r1, 2.0 * r1))
        off += n * dim
    return descs, off


def _ridge_and_ideal(case, seed):
    """A finished ridge (points along the helix, somewhat off it) and the ideal curve's points."""
    g = _generator(seed)
    t = torch.linspace(0.0, 8.0 * math.pi, case["n"], device="cuda", dtype=torch.float64)
    t = t[torch.randperm(case["n"], generator=g, device="cuda")]
    S = torch.stack([torch.cos(t), torch.sin(t), 0.15 * t], 1) + _normal(g, (case["n"], 3), 0.01)
    u = _uniform(g, case["ideal"], 0.0, 8.0 * math.pi)
    ideal = torch.stack([torch.cos(u), torch.sin(u), 0.15 * u], 1)
    return S.float().contiguous(), ideal.float().contiguous()


def _adjoint_inputs(case, seed):
    P = _helix(_generator(seed), case["n"]).float().contiguous()
    S0 = _greedy(P, case["r1"])
    # the chosen points are points of the cloud: the first that equals each
    idx = torch.stack([(P == s).all(1).nonzero()[0, 0] for s in S0])
    w = torch.randn(S0.shape, generator=_generator(seed + 1), device="cuda", dtype=torch.float32)
    return P, idx, w


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind == "solve":
        P = _cloud(case, seed)
        if case["layout"] == "col":
            P = P.t().contiguous()
        s["P"] = P.cpu().numpy() if case["host"] else P
        layout = rdb.COL_MAJOR if case["layout"] == "col" else rdb.ROW_MAJOR
        dim = 2 if case["gen"] == "sine" else 3
        s["h"] = rdb.BruteForceRidgeDetection(case["n"], case["r1"], case["r2"], dim,
                                              in_layout=layout, out_layout=layout)
        s["out"] = np.zeros((dim, RIDGE_ROWS) if case["layout"] == "col" else (RIDGE_ROWS, dim),
                            np.float32)
        s["pitch"] = RIDGE_ROWS if case["layout"] == "col" else dim
    elif kind == "tiled":
        s["P"] = _spiral(_generator(seed), case["n"], 0.05).float().contiguous()
        s["h"] = rdb.TiledRidgeDetection(case["n"], 2)
        s["out"] = np.zeros((CHOSEN_ROWS, 2), np.float32)
    elif kind == "batch":
        s["descs"], total = _batch_descs(case)
        g = _generator(seed)
        s["P"] = torch.empty(total, device="cuda", dtype=torch.float32)
        for off, n, dim, _, _ in s["descs"]:
            p = _sine(g, n) if dim == 2 else _helix(g, n)
            s["P"][off:off + n * dim] = p.reshape(-1).float()
        s["h"] = rdb.BatchedRidgeDetection()
        s["out"] = np.zeros((case["clouds"], RIDGE_ROWS, 3), np.float32)
    elif kind == "choose":
        s["P"] = _cloud(case, seed)
        s["S"] = torch.zeros_like(s["P"])
    elif kind == "evolve":
        s["P"] = _cloud(case, seed)
        s["S0"] = _greedy(s["P"], case["r1"])
        s["S"] = torch.zeros((CHOSEN_ROWS, s["P"].shape[1]), device="cuda")
    elif kind == "decimate":
        s["S0"] = _spiral(_generator(seed), case["n"], 0.0).float().contiguous()
    elif kind == "adjoint":
        s["P"], s["idx"], s["w"] = _adjoint_inputs(case, seed)
        s["P"].requires_grad_(True)
        s["f"] = evolve_function()
        s["S"] = torch.zeros((CHOSEN_ROWS, 3), device="cuda")
    else:
        s["S"], s["I"] = _ridge_and_ideal(case, seed)
        s["chains"] = np.zeros(case["n"] + 1, np.int32)
    return s


# --- one pass -------------------------------------------------------------------------------------

def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def run(s):
    kind = s["kind"]
    if kind == "solve":
        s["h"].set_points(s["P"])
        s["h"].ridge_detection()
        return {"S": s["h"].chosen_points(s["out"], s["pitch"]), "count": s["h"].ns_}
    if kind == "tiled":
        s["h"].set_points(s["P"])
        s["h"](s["r1"], s["r2"], s["capacity"], (s["tiles"], s["tiles"]))
        return {"S": s["h"].get_chosen_points(s["out"]), "count": s["h"].ns_}
    if kind == "batch":
        counts = s["h"].run(s["P"], s["descs"])
        for c, (_, _, dim, _, _) in enumerate(s["descs"]):
            s["out"][c, :counts[c], :dim] = s["h"].chosen_points(c)
        return {"counts": counts, "S": s["out"]}
    lib = rdb.lib()
    if kind == "choose":
        n, dim = s["P"].shape
        ns = ctypes.c_int64(0)
        L.check(lib.rd_choose(dim, _ptr(s["P"]), n, s["r1"], _ptr(s["S"]), ctypes.byref(ns),
                              _stream()))
        return {"S": s["S"], "count": ns.value}
    if kind == "evolve":
        n, dim = s["P"].shape
        ns = s["S0"].shape[0]
        s["S"][:ns].copy_(s["S0"])
        moved = ctypes.c_int32(0)
        L.check(lib.rd_evolve_pass(dim, _ptr(s["P"]), n, _ptr(s["S"]), ns, s["r1"],
                                   ctypes.byref(moved), _stream()))
        return {"S": s["S"], "moved": moved.value}
    if kind == "decimate":
        S = s["S0"].clone()
        left = ctypes.c_int64(0)
        L.check(lib.rd_decimate(S.shape[1], _ptr(S), S.shape[0], s["r2"], ctypes.byref(left),
                                _stream()))
        return {"S": S, "count": left.value}
    if kind == "adjoint":
        s["P"].grad = None
        S = s["f"].apply(s["P"], s["idx"], s["r1"], s["iters"], s["every"])
        (S * s["w"]).sum().backward()
        s["S"][:S.shape[0]].copy_(S.detach())
        return {"S": s["S"], "grad": s["P"].grad}
    order, chains = rdb.order_chains(s["S"], s["r2"])
    s["chains"][:chains.shape[0]] = chains
    return {"order": order, "chains": s["chains"], "hausdorff": rdb.hausdorff(s["S"], s["I"]),
            "stats": list(rdb.distance_stats(s["S"], s["I"]))}


# --- what one pass cannot do without --------------------------------------------------------------

def work(case):
    """Inputs read once and outputs written once.  A solve's number of passes depends on its cloud;
    counted is one distance per point, so a solve's figure is that of its first pass at best."""
    kind = case["kind"]
    if kind == "batch":
        descs, floats = _batch_descs(case)
        return {"bytes": 4 * floats, "flops": 3 * floats}
    if kind == "report":
        pairs = case["n"] * case["ideal"]
        return {"bytes": 12 * (case["n"] + case["ideal"]), "flops": 3 * 3 * 3 * pairs}
    dim = 2 if kind in ("tiled", "decimate") or case.get("gen") == "sine" else 3
    cloud = 4 * dim * case["n"]
    if kind == "adjoint":
        return {"bytes": 2 * cloud, "flops": 3 * dim * case["n"] * case["iters"]}
    return {"bytes": cloud, "flops": 3 * dim * case["n"]}


# --- the same in 64 bits --------------------------------------------------------------------------

def _rows(S, n):
    return torch.nn.functional.pad(S, (0, 0, 0, n - S.shape[0]))


def _assign64(P, S, r1):
    """Index of the nearest chosen point of each cloud point, -1 where it is further than r1."""
    r1 = torch.tensor(r1, dtype=torch.float32).item()
    step = max(1, 40_000_000 // S.shape[0])
    out = []
    for p in P.split(step):
        d2 = torch.zeros((p.shape[0], S.shape[0]), device=P.device, dtype=torch.float64)
        for d in range(P.shape[1]):
            t = p[:, d, None] - S[None, :, d]
            d2 += t * t
        v, k = d2.min(1)
        out.append(torch.where(v <= r1 * r1, k, torch.full_like(k, -1)))
    return torch.cat(out)


def _pass64(P, S, r1):
    """(new chosen points, members per chosen point, key of each point)"""
    key = _assign64(P, S, r1)
    at = key >= 0
    cnt = torch.bincount(key[at], minlength=S.shape[0]).double()
    total = torch.zeros_like(S).index_add_(0, key[at], P[at])
    mean = torch.where(cnt[:, None] > 0, total / cnt.clamp(min=1)[:, None], S)
    return mean, cnt, key


def exact(case, seed):
    kind = case["kind"]
    if kind == "choose":
        return {"S": _rows(_greedy(_cloud(case, seed).double(), case["r1"]), case["n"]),
                "count": None}
    if kind == "evolve":
        P = _cloud(case, seed)
        S = _pass64(P.double(), _greedy(P, case["r1"]).double(), case["r1"])[0]
        return {"S": _rows(S, CHOSEN_ROWS), "moved": None}
    if kind == "adjoint":
        P, idx, w = _adjoint_inputs(case, seed)
        P, S, g = P.double(), P.double()[idx], w.double()
        passes = []
        for _ in range(case["iters"]):
            S, cnt, key = _pass64(P, S, case["r1"])
            passes.append((cnt, key))
        grad = torch.zeros_like(P)
        for cnt, key in reversed(passes):
            at = key >= 0
            grad[at] += (g / cnt.clamp(min=1)[:, None])[key[at]]
            g = torch.where(cnt[:, None] > 0, torch.zeros_like(g), g)
        grad.index_add_(0, idx, g)
        return {"S": _rows(S, CHOSEN_ROWS), "grad": grad}
    if kind == "report":
        S, ideal = (x.double() for x in _ridge_and_ideal(case, seed))
        d = torch.cdist(S, ideal, compute_mode="donot_use_mm_for_euclid_dist")
        near = d.amin(1).sort().values
        median = near[near.shape[0] // 2]
        return {"order": None, "chains": None,
                "hausdorff": float(max(near[-1], d.amin(0).max())),
                "stats": [float(median), float(near.mean()), float(near[0]), float(near[-1])]}
    # a whole solve, a decimation: points kept or moved by many threshold decisions in 32 bits
    return None

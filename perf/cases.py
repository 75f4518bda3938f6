"""The work that users of this framework have it do, as cases that can be timed.

Every case goes through a public entry point of ``rtdsl``: the captured and
the eager k_nn! pipelines, searches on a kept index, the host-buffer k_nn!,
the differentiable k-NN, the range query, DBSCAN, the batched clouds, and
Barnes-Hut with its adjoint, its leapfrog and its reference law.  Sizes come
from the workloads of rtdsl/workloads.py, bench.py and tests/; inputs follow
the same distributions, drawn on the GPU.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("rt-dsl_b200"))
import rtdsl  # noqa: E402
from rtdsl import torch_ops  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # The smallest call: a few thousand points that change on every call
        # (an interactive tool, the smoke test's size); latency and launches.
        {"name": "call_2k", "kind": "call", "dist": "uniform", "n": 2003, "nq": 509, "k": 5},
        # k_nn!(data, queries, k, out) as the macro's users write it: host
        # arrays in and out, the plain_knn_small workload.
        {"name": "host_100k", "kind": "host", "dist": "uniform", "n": 100_000, "nq": 10_000, "k": 5},
        # The headline: the whole pipeline replayed per frame on new contents
        # of fixed buffers, clustered_1p8m with its tuned schedule.
        {"name": "graph_1p8m", "kind": "graph", "dist": "clustered", "n": 1_800_000, "nq": 400_000, "k": 5},
        # The largest cloud: build and search of the dense sheet_10m.
        {"name": "sheet_10m", "kind": "sheet", "dist": "sheet", "n": 10_000_000, "nq": 1_000_000, "k": 16},
        # New queries against an index that stays, with a long neighbour list
        # (graph construction, density estimates).
        {"name": "search_k300", "kind": "search", "dist": "clustered", "n": 1_800_000, "nq": 40_000, "k": 300},
        # A training step on k-NN distances: forward and backward through
        # autograd on points that moved since the last step.
        {"name": "train_50k", "kind": "train", "dist": "clustered", "n": 50_021, "nq": 50_021, "k": 16},
        # range_query! on device buffers: build, count, and the pairs sorted
        # by (query, id), 50 neighbours a query.
        {"name": "range_1p8m", "kind": "range", "dist": "clustered", "n": 1_800_000, "nq": 400_000, "mean": 50},
        # DBSCAN with 20 mean neighbours, min_pts 10.
        {"name": "dbscan_200k", "kind": "dbscan", "dist": "clustered", "n": 200_000, "mean": 20, "min_pts": 10},
        # Many clouds of uneven size with k of their own, forward and
        # backward: the clouds_256 workload.
        {"name": "clouds_256", "kind": "batch", "clouds": 256, "lo": 1000, "hi": 200_000},
        # A differentiable N-body step: build, forces and potentials, adjoint;
        # the plummer_1m workload.
        {"name": "bh_grad_1m", "kind": "bh_grad", "n": 1_000_000, "theta": 0.5, "bucket": 32, "quad": 1},
        # Time integration: four leapfrog steps, the tree rebuilt in each.
        {"name": "leapfrog_100k", "kind": "leapfrog", "n": 100_003, "theta": 0.5, "bucket": 32, "steps": 4},
        # barnes_hut!(bodies, theta, G, out): host bodies, the reference law.
        {"name": "reference_bh_50k", "kind": "reference", "n": 50_000, "theta": 0.5},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "host", "graph", "sheet", "search", "train", "range", "dbscan", "batch",
                       "bh_grad", "leapfrog", "reference"])
    dist = rng.choice(["uniform", "clustered"])
    if kind == "call":
        n = _log(rng, 700, 150_000)
        return {"kind": kind, "dist": dist, "n": n, "nq": _log(rng, 100, n), "k": rng.choice([1, 3, 5, 8, 16])}
    if kind == "host":
        n = _log(rng, 20_000, 1_000_000)
        return {"kind": kind, "dist": dist, "n": n, "nq": _log(rng, 2_000, n // 4), "k": rng.choice([1, 5, 8, 16])}
    if kind == "graph":
        n = _log(rng, 200_000, 1_800_000)
        return {"kind": kind, "dist": "clustered", "n": n, "nq": _log(rng, 20_000, 400_000), "k": rng.randint(1, 8)}
    if kind == "sheet":
        return {"kind": kind, "dist": "sheet", "n": _log(rng, 700_000, 10_000_000),
                "nq": _log(rng, 70_000, 1_000_000), "k": rng.choice([1, 5, 10, 16])}
    if kind == "search":
        return {"kind": kind, "dist": dist, "n": _log(rng, 100_000, 1_800_000), "nq": _log(rng, 2_000, 40_000),
                "k": _log(rng, 17, 1000)}
    if kind == "train":
        n = _log(rng, 8_000, 200_000)
        return {"kind": kind, "dist": dist, "n": n, "nq": _log(rng, 4_000, n), "k": rng.randint(3, 16)}
    if kind == "range":
        return {"kind": kind, "dist": dist, "n": _log(rng, 50_000, 1_800_000), "nq": _log(rng, 20_000, 400_000),
                "mean": _log(rng, 8, 60)}
    if kind == "dbscan":
        return {"kind": kind, "dist": "clustered", "n": _log(rng, 30_000, 1_800_000), "mean": rng.randint(8, 24),
                "min_pts": rng.randint(4, 12)}
    if kind == "batch":
        return {"kind": kind, "clouds": _log(rng, 12, 256), "lo": 1000, "hi": _log(rng, 8_000, 200_000)}
    if kind == "bh_grad":
        return {"kind": kind, "n": _log(rng, 16_000, 1_000_000), "theta": rng.choice([0.5, 0.6, 0.75, 0.9]),
                "bucket": rng.choice([16, 32]), "quad": rng.choice([0, 1])}
    if kind == "leapfrog":
        return {"kind": kind, "n": _log(rng, 10_000, 500_000), "theta": rng.choice([0.5, 0.7]), "bucket": 32,
                "steps": rng.randint(1, 4)}
    return {"kind": kind, "n": _log(rng, 2_000, 200_000), "theta": rng.choice([0.5, 0.8])}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _jittered(g, pts, nq, sigma):
    sel = torch.randint(0, pts.shape[0], (nq,), generator=g, device=DEV)
    return (pts[sel] + torch.randn((nq, 3), generator=g, device=DEV) * sigma).contiguous()


def _uniform(g, n, nq):
    pts = torch.rand((n, 3), generator=g, device=DEV)
    return pts, _jittered(g, pts, nq, 1e-3)


def _clustered(g, n, nq, n_clusters=64, box=100.0):
    """90 % of the points from anisotropic Gaussians, 10 % uniform."""
    centres = torch.rand((n_clusters, 3), generator=g, device=DEV) * box
    sigma = torch.exp(torch.rand((n_clusters, 3), generator=g, device=DEV) * math.log(100.0) + math.log(0.05))
    lab = torch.randint(0, n_clusters, (n,), generator=g, device=DEV)
    pts = centres[lab] + torch.randn((n, 3), generator=g, device=DEV) * sigma[lab]
    background = torch.rand((n,), generator=g, device=DEV) < 0.1
    pts = torch.where(background[:, None], torch.rand((n, 3), generator=g, device=DEV) * box, pts).contiguous()
    return pts, _jittered(g, pts, nq, 0.01)


def _sheet(g, n, nq, n_hot=2000):
    """Zipf-weighted hotspots of a thin sheet."""
    centres = torch.rand((n_hot, 2), generator=g, device=DEV) * 10.0
    sigma = torch.exp(torch.rand((n_hot,), generator=g, device=DEV) * math.log(100.0) + math.log(1e-3))
    w = 1.0 / torch.arange(1, n_hot + 1, device=DEV) ** 1.2

    def sample(m):
        lab = torch.multinomial(w, m, replacement=True, generator=g)
        xy = centres[lab] + torch.randn((m, 2), generator=g, device=DEV) * sigma[lab, None]
        z = torch.randn((m, 1), generator=g, device=DEV) * 1e-4
        return torch.cat([xy.clamp_(0.0, 10.0), z], 1).contiguous()

    return sample(n), sample(nq)


def _points(case, g):
    make = {"uniform": _uniform, "clustered": _clustered, "sheet": _sheet}[case["dist"]]
    return make(g, case["n"], case.get("nq", 1))


def _plummer(g, n):
    """Plummer sphere, scale radius 1, total mass 1, equal masses."""
    x = torch.rand((n,), generator=g, device=DEV, dtype=torch.float64).clamp_(1e-6, 1.0 - 1e-6)
    r = 1.0 / torch.sqrt(x ** (-2.0 / 3.0) - 1.0)
    cz = torch.rand((n,), generator=g, device=DEV, dtype=torch.float64) * 2.0 - 1.0
    ph = torch.rand((n,), generator=g, device=DEV, dtype=torch.float64) * (2.0 * math.pi)
    sz = torch.sqrt(1.0 - cz * cz)
    pos = torch.stack([r * sz * torch.cos(ph), r * sz * torch.sin(ph), r * cz], 1)
    return pos.float().contiguous(), torch.full((n,), 1.0 / n, device=DEV)


def _radius(pts, queries, mean):
    """Radius of about `mean` neighbours a query, from a sample of both sets."""
    q = queries[:: max(1, queries.shape[0] // 512)][:512]
    p = pts[:: max(1, pts.shape[0] // 65536)]
    d = torch.sort(torch.cdist(q, p, compute_mode="donot_use_mm_for_euclid_dist").reshape(-1))[0]
    at = int(mean * q.shape[0] * p.shape[0] / pts.shape[0])
    return float(d[min(max(at, 1), d.numel() - 1)])


def _cloud_sizes(case):
    """(points, queries, k) of every cloud; the same for every seed."""
    r = random.Random(case["clouds"] * 1_000_003 + case["hi"])
    sizes = [_log(r, case["lo"], case["hi"]) for _ in range(case["clouds"])]
    return [(n, max(1, n // 4), r.choice([1, 5, 16, 64])) for n in sizes]


def _clouds(case, g):
    """Alternately uniform clouds and mixtures of eight Gaussians in the unit cube."""
    pts, qs = [], []
    for c, (n, nq, _) in enumerate(_cloud_sizes(case)):
        p = torch.rand((n, 3), generator=g, device=DEV)
        if c % 2:
            cen = torch.rand((8, 3), generator=g, device=DEV) * 0.8 + 0.1
            sg = torch.rand((8, 1), generator=g, device=DEV) * 0.07 + 0.01
            lab = torch.randint(0, 8, (n,), generator=g, device=DEV)
            p = (cen[lab] + torch.randn((n, 3), generator=g, device=DEV) * sg[lab]).clamp_(0.0, 1.0)
        pts.append(p)
        qs.append(_jittered(g, p, nq, 1e-3).clamp_(0.0, 1.0))
    return torch.cat(pts).contiguous(), torch.cat(qs).contiguous()


def _bh_params(case):
    return rtdsl.default_bh_params(law=rtdsl.BH_LAW_PLUMMER, theta=case["theta"], eps=1e-3, G=1.0,
                                   quadrupole=case.get("quad", 1), bucket=case["bucket"])


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    s = {"case": case}
    if kind in ("bh_grad", "leapfrog", "reference"):
        s["pos"], s["mass"] = _plummer(g, case["n"])
        if kind == "reference":
            s["bodies"] = torch.cat([s["pos"], s["mass"][:, None]], 1).cpu().numpy()
            return s
        s["params"], s["bh"] = _bh_params(case), rtdsl.BarnesHut()
        if kind == "bh_grad":
            s["g_acc"] = torch.randn((case["n"], 3), generator=g, device=DEV)
            s["g_phi"] = torch.randn((case["n"],), generator=g, device=DEV)
        else:
            s["vel"] = torch.randn((case["n"], 3), generator=g, device=DEV) * 0.3
        return s
    if kind == "batch":
        s["points"], s["queries"] = _clouds(case, g)
        s["batch"] = rtdsl.Batch(_cloud_sizes(case))
        s["g_d2"] = torch.randn((s["batch"].n_out,), generator=g, device=DEV)
        return s
    s["points"], s["queries"] = _points(case, g)
    if kind == "call":
        s["index"] = rtdsl.Index()
    elif kind == "host":
        s["points"], s["queries"] = s["points"].cpu().numpy(), s["queries"].cpu().numpy()
    elif kind == "graph":
        tuned = rtdsl.default_schedule(radius_heuristic=rtdsl.RADIUS_MORTON_WINDOW, radius_param=0.5, leaf_size=5,
                                       morton_bits=39, block_size=128, lanes_per_query=1)
        s["graph"] = rtdsl.KnnGraph(s["points"], s["queries"], case["k"], tuned)
    elif kind == "sheet":
        s["index"] = rtdsl.Index()
    elif kind == "search":
        s["index"] = rtdsl.Index().build(s["points"])
    elif kind == "train":
        s["points"].requires_grad_()
        s["queries"].requires_grad_()
        s["g_d2"] = torch.randn((case["nq"], case["k"]), generator=g, device=DEV)
    else:
        if kind == "dbscan":
            s["queries"] = s["points"]
        s["radius"] = _radius(s["points"], s["queries"], case["mean"])
        s["index"] = rtdsl.Index()
        s["schedule"] = rtdsl.default_schedule(leaf_size=12, morton_bits=42)
        if kind == "range":   # a pair buffer kept between calls, with room to spare
            s["pairs"] = torch.zeros((2 * case["nq"] * case["mean"] + 65536, 2), dtype=torch.int32, device=DEV)
    return s


# -------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "call":
        return s["index"].k_nn(s["points"], s["queries"], case["k"])
    if kind == "host":
        return rtdsl.k_nn_array(s["points"], s["queries"], case["k"])
    if kind == "graph":
        return s["graph"].launch()
    if kind == "sheet":
        return s["index"].build(s["points"]).knn(s["queries"], case["k"])
    if kind == "search":
        return s["index"].knn(s["queries"], case["k"])
    if kind == "train":
        d2, ids = torch_ops.knn_distances(s["queries"], s["points"], case["k"])
        g_q, g_p = torch.autograd.grad(d2, (s["queries"], s["points"]), s["g_d2"])
        return d2.detach(), ids, g_q, g_p
    if kind == "range":
        ix, q, r, sched = s["index"], s["queries"], s["radius"], s["schedule"]
        ix.build(s["points"], sched)
        counts, total = ix.range_count(q, r, sched)
        buf = s["pairs"]
        ix.range_fill(q, r, buf.shape[0], sort_pairs=True, schedule=sched, out_pairs=buf)
        return counts, total, buf
    if kind == "dbscan":
        s["index"].build(s["points"], s["schedule"])
        return rtdsl.dbscan(s["points"], s["radius"], case["min_pts"], index=s["index"])
    if kind == "batch":
        b = s["batch"]
        ids, d2 = b.knn(s["points"], s["queries"])
        g_q, g_p = b.backward(s["points"], s["queries"], ids, s["g_d2"])
        return ids, d2, g_q, g_p
    if kind == "bh_grad":
        bh, p = s["bh"], s["params"]
        bh.build(s["pos"], s["mass"], p)
        acc, phi = bh.forward(p)
        g_pos, g_mass = bh.backward(s["g_acc"], s["g_phi"], p)
        return acc, phi, g_pos, g_mass
    if kind == "leapfrog":
        pos, vel = s["pos"].clone(), s["vel"].clone()
        acc = s["bh"].leapfrog(pos, vel, s["mass"], 1e-3, case["steps"], s["params"])
        return pos, vel, acc
    return rtdsl.barnes_hut(s["bodies"], case["theta"], G=1.0)


def work(case):
    """What a pass cannot do without: its inputs and outputs once, and for the
    N-body sums the arithmetic of one interaction per accepted cell and
    near body (counts of the Plummer sphere, measured; they grow with log n
    and shrink with theta)."""
    kind, n = case["kind"], case.get("n", 0)
    if kind in ("bh_grad", "leapfrog", "reference"):
        pairs = n * (240.0 * math.log2(n) - 1450.0) * (0.5 / case["theta"]) ** 2.25
        if kind == "bh_grad":
            return {"bytes": n * (16 + 16 + 16 + 16), "flops": pairs * 120}
        if kind == "leapfrog":
            return {"bytes": n * (28 + 36), "flops": pairs * 40 * (case["steps"] + 1)}
        return {"bytes": n * 28, "flops": pairs * 25}
    if kind == "batch":
        sizes = _cloud_sizes(case)
        np_, nq, out = sum(x[0] for x in sizes), sum(x[1] for x in sizes), sum(x[1] * x[2] for x in sizes)
        return {"bytes": 12 * (np_ + nq) + 8 * out + 4 * out + 12 * (np_ + nq), "flops": 0}
    nq = case.get("nq", n)
    if kind == "range":
        return {"bytes": 12 * (n + nq) + 4 * nq + 8 * nq * case["mean"], "flops": 0}
    if kind == "dbscan":
        return {"bytes": 16 * n, "flops": 0}
    k = case["k"]
    rw = 12 * (n + nq) + 8 * k * nq
    return {"bytes": rw + (4 * k * nq + 12 * (n + nq) if kind == "train" else 0), "flops": 0}


# ------------------------------------------------------- 64-bit values
def _exact_knn(pts, q, k):
    """Squared distances of the k nearest (64-bit), ascending, and their points."""
    p, q = pts.double(), q.double()
    rows = max(1, 60_000_000 // p.shape[0])
    d2s, ids = [], []
    for c in q.split(rows):
        d = (c[:, None, 0] - p[None, :, 0]).square_()
        d += (c[:, None, 1] - p[None, :, 1]).square_()
        d += (c[:, None, 2] - p[None, :, 2]).square_()
        v, i = torch.topk(d, min(k, p.shape[0]), largest=False, sorted=True)
        d2s.append(v)
        ids.append(i)
    return torch.cat(d2s), torch.cat(ids)


def _exact_knn_grad(pts, q, ids, g):
    diff = q.double()[:, None, :] - pts.double()[ids]
    w = 2.0 * g.double()[:, :, None] * diff
    gp = torch.zeros(pts.shape, dtype=torch.float64, device=pts.device)
    gp.index_add_(0, ids.reshape(-1), -w.reshape(-1, 3))
    return w.sum(1), gp


def _direct(pos, mass, g_acc=None, g_phi=None):
    """Plummer accelerations and potentials of every pair, and the gradients
    of sum(g_acc . acc) + sum(g_phi phi)."""
    x = pos.double().requires_grad_(g_acc is not None)
    m = mass.double().requires_grad_(g_acc is not None)
    n = x.shape[0]
    acc, phi = torch.empty((n, 3), dtype=torch.float64, device=DEV), torch.empty((n,), dtype=torch.float64, device=DEV)
    step = max(1, 12_000_000 // n)
    for a in range(0, n, step):
        b = min(n, a + step)
        d = x[None, :, :] - x[a:b, None, :]
        inv = torch.rsqrt(d.square().sum(2) + 1e-6)
        own = torch.zeros_like(inv, requires_grad=False)
        own[torch.arange(b - a, device=DEV), torch.arange(a, b, device=DEV)] = 1.0
        w = m[None, :] * inv * (1.0 - own)
        p, f = -w.sum(1), torch.einsum("ij,ijc->ic", w * inv * inv, d)
        if g_acc is not None:
            ((f * g_acc[a:b].double()).sum() + (p * g_phi[a:b].double()).sum()).backward()
        acc[a:b], phi[a:b] = f.detach(), p.detach()
    return acc, phi, x.grad, m.grad


def _direct_reference(pos, mass, G):
    """The reference law over every pair."""
    x, m = pos.double(), mass.double()
    out, step = torch.empty_like(x), max(1, 12_000_000 // x.shape[0])
    for a in range(0, x.shape[0], step):
        d = x[None, :, :] - x[a:a + step, None, :]
        r2 = d.square().sum(2)
        w = torch.where(r2 > 1e-10, G * m[a:a + step, None] * m[None, :] / (r2 * torch.sqrt(r2 + 1e-6)), 0.0)
        out[a:a + step] = torch.einsum("ij,ijc->ic", w, d)
    return out


def exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    if kind in ("range", "dbscan"):
        return None   # whole numbers only
    g = _gen(seed)
    if kind in ("bh_grad", "leapfrog", "reference"):
        if n > 120_000:
            return None
        pos, mass = _plummer(g, n)
        if kind == "reference":
            return _direct_reference(pos, mass, 1.0)
        if kind == "bh_grad":
            g_acc = torch.randn((n, 3), generator=g, device=DEV)
            g_phi = torch.randn((n,), generator=g, device=DEV)
            return _direct(pos, mass, g_acc, g_phi)
        x, v = pos.double(), (torch.randn((n, 3), generator=g, device=DEV) * 0.3).double()
        acc = _direct(x, mass)[0]
        for _ in range(case["steps"]):
            v = v + acc * 0.5e-3
            x = x + v * 1e-3
            acc = _direct(x, mass)[0]
            v = v + acc * 0.5e-3
        return x, v, acc
    if kind == "batch":
        sizes = _cloud_sizes(case)
        if sum(a * b for a, b, _ in sizes) > 1.5e10:
            return None
        pts, q = _clouds(case, g)
        g_d2 = torch.randn((sum(b * k for _, b, k in sizes),), generator=g, device=DEV)
        d2, gq, gp = [], [], []
        po = qo = oo = 0
        for a, b, k in sizes:
            p1, q1, g1 = pts[po:po + a], q[qo:qo + b], g_d2[oo:oo + b * k].reshape(b, k)
            d, i = _exact_knn(p1, q1, k)
            x, y = _exact_knn_grad(p1, q1, i, g1)
            d2.append(d.reshape(-1))
            gq.append(x)
            gp.append(y)
            po, qo, oo = po + a, qo + b, oo + b * k
        return None, torch.cat(d2), torch.cat(gq), torch.cat(gp)
    if n * case["nq"] > 1.5e10:
        return None
    pts, q = _points(case, g)
    d2, ids = _exact_knn(pts, q, case["k"])
    if kind == "train":
        g_d2 = torch.randn((case["nq"], case["k"]), generator=g, device=DEV)
        return (d2, None) + _exact_knn_grad(pts, q, ids, g_d2)
    return None, d2

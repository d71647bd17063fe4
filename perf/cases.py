"""The work that users of this package have it do, as cases that can be timed
and compared: whole triangulations from a few hundred points to eight million,
on the device (torch CUDA tensors in and out) and through the numpy API, the
batched call, the scheduler and ordering options, and the check of a finished
triangulation.

A triangulation numbers its tets in the order in which the insertion rounds
left them, which differs from run to run; the canonical form (ids sorted in
each row, rows sorted, adjacency re-indexed) is unique.  So a pass here is the
triangulation followed by its canonical form, as a program does that stores,
compares or digests its results, kept in arrays of a fixed number of rows (the
library's bound wtet_max_tets, the rest filled).

A case: `task` ("triangulate", "batch", "verify"), `where` the data live
("device", "host"), `cloud` the distribution, `n` the points (`batch`: `clouds`
clouds with sizes log-uniform in [lo, hi]; `lattice`: `n` sites per axis), and
the Config options `vote`, `rule`, `hilbert`.
"""
import math

import numpy as np
import torch

import wtet_b200 as wt


def _case(name, task, where, cloud, n, vote="plain", rule="circumcenter", hilbert=False):
    c = {"task": task, "where": where, "cloud": cloud, "n": n, "vote": vote, "rule": rule, "hilbert": hilbert}
    return dict(c, name=name) if name else c


def _batch(name, clouds, lo, hi):
    c = {"task": "batch", "where": "host", "cloud": "batch", "clouds": clouds, "lo": lo, "hi": hi,
         "vote": "plain", "rule": "circumcenter", "hilbert": False}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one small object (a molecule, a cell's neighbourhood) per call from a device-resident loop: latency alone
        _case("dev_uniform_200", "triangulate", "device", "uniform", 200),
        # the package's first example: a thousand numpy points, result back in numpy
        _case("host_uniform_1000", "triangulate", "host", "uniform", 1000),
        # a scan's worth of clustered points with the Hilbert order and the centroid rule
        _case("dev_clustered_20011_hilbert", "triangulate", "device", "clustered", 20011, rule="centroid",
              hilbert=True),
        # the small configuration of the benchmark
        _case("dev_uniform_100k", "triangulate", "device", "uniform", 100_000),
        # surface samples: every point on the unit sphere (no points inside)
        _case("dev_sphere_250k", "triangulate", "device", "sphere", 250_000),
        # vertices of a voxel grid with a tenth of the sites masked out: cospherical and coplanar everywhere
        _case("dev_lattice_72", "triangulate", "device", "lattice", 72),
        # a million points of the benchmark's mixture, plain and with the learned scheduler
        _case("dev_mixture_1M", "triangulate", "device", "mixture", 1_000_000),
        _case("dev_mixture_1M_learned", "triangulate", "device", "mixture", 1_000_000, vote="learned"),
        # the same order of size through the numpy API: upload, triangulation, download
        _case("host_uniform_700k", "triangulate", "host", "uniform", 700_001),
        # many clouds of uneven sizes in one call (the batched configuration's distribution)
        _batch("host_batch_256", 256, 64, 65536),
        # the exact check of a stored triangulation
        _case("dev_verify_1M", "verify", "device", "mixture", 1_000_000),
        # the benchmark's headline
        _case("dev_mixture_8M", "triangulate", "device", "mixture", 8_000_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.randrange(8)
    if kind == 0:  # small device calls
        return _case(None, "triangulate", "device", rng.choice(["uniform", "clustered", "mixture"]),
                     _log(rng, 64, 4000), rule=rng.choice(["circumcenter", "centroid"]))
    if kind == 1:  # numpy calls
        return _case(None, "triangulate", "host", rng.choice(["uniform", "clustered"]), _log(rng, 100, 800_000))
    if kind == 2:  # ordinary sizes, either order and rule
        return _case(None, "triangulate", "device", rng.choice(["uniform", "mixture", "clustered"]),
                     _log(rng, 4000, 200_000), rule=rng.choice(["circumcenter", "centroid"]),
                     hilbert=rng.random() < 0.5)
    if kind == 3:
        return _case(None, "triangulate", "device", "sphere", _log(rng, 2000, 300_000))
    if kind == 4:
        return _case(None, "triangulate", "device", "lattice", rng.randrange(9, 81))
    if kind == 5:  # large ones, both schedulers
        return _case(None, "triangulate", "device", rng.choice(["uniform", "mixture"]), _log(rng, 200_000, 8_000_000),
                     vote=rng.choice(["plain", "learned"]))
    if kind == 6:
        lo = _log(rng, 32, 1000)
        return _batch(None, _log(rng, 8, 300), lo, lo * rng.randrange(2, 65))
    return _case(None, "verify", "device", rng.choice(["uniform", "mixture"]), _log(rng, 1000, 1_000_000))


def _points(cloud, n):
    """Points of a cloud: nine tenths of the sites of a lattice with n sites per axis, else n."""
    return n ** 3 - n ** 3 // 10 if cloud == "lattice" else n


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _directions(m, g):
    d = torch.randn((m, 3), generator=g, device="cuda", dtype=torch.float64)
    return d / d.norm(dim=1, keepdim=True)


def _cloud(kind, n, g):
    """One cloud as a CUDA float32 tensor (the distributions of wtet_b200.synthetic, drawn on the device)."""
    rand = lambda *s: torch.rand(s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    randn = lambda *s: torch.randn(s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    if kind == "uniform":
        p = rand(n, 3)
    elif kind == "mixture":
        nu, ng = round(0.6 * n), round(0.3 * n)
        ns = n - nu - ng
        p = torch.cat([rand(nu, 3), 0.5 + 0.1 * randn(ng, 3),
                       0.5 + (0.4 + 1e-4 * randn(ns, 1)) * _directions(ns, g)])
        p = p[torch.randperm(n, generator=g, device="cuda")]
    elif kind == "clustered":
        centers = rand(8, 3) * 0.8 + 0.1
        which = torch.randint(0, 8, (n,), generator=g, device="cuda")
        p = centers[which] + 0.05 * randn(n, 3)
    elif kind == "gauss":
        p = 0.5 + 0.1 * randn(n, 3)
    elif kind == "shell":
        p = 0.5 + (0.4 + 1e-4 * randn(n, 1)) * _directions(n, g)
    elif kind == "sphere":
        p = _directions(n, g)
    elif kind == "jittered":
        m = math.ceil(n ** (1.0 / 3.0))
        i = torch.arange(n, device="cuda")
        p = torch.stack([i // (m * m), i // m % m, i % m], 1).double() / m + 1e-6 * (2.0 * rand(n, 3) - 1.0)
    else:  # lattice: n sites per axis in raster order, a tenth masked out
        i = torch.randperm(n ** 3, generator=g, device="cuda")[: _points("lattice", n)].sort().values
        c = (torch.arange(n, device="cuda", dtype=torch.float32) / (n - 1))
        p = torch.stack([c[i // (n * n)], c[i // n % n], c[i % n]], 1)
    return p.to(torch.float32).contiguous()


def _sizes(case):
    """Sizes of a batch's clouds: the quantiles of a log-uniform law, in a fixed shuffled order."""
    q = (np.arange(case["clouds"]) + 0.5) / case["clouds"]
    sizes = np.floor(np.exp(math.log(case["lo"]) + q * math.log(case["hi"] / case["lo"]))).astype(np.int64)
    return np.random.default_rng(case["clouds"]).permutation(sizes)


def _batch_clouds(case, seed):
    kinds = np.random.default_rng(seed).integers(0, 4, case["clouds"])
    g = _gen(seed)
    return [_cloud(("uniform", "gauss", "shell", "jittered")[k], int(n), g).cpu().numpy()
            for n, k in zip(_sizes(case), kinds)]


def _max_tets(n):
    return 8 * int(n) + 64


def prepare(case, seed):
    cfg = wt.Config(vote=case["vote"], insertion_rule=case["rule"], enable_hilbert_sorting=case["hilbert"])
    state = {"task": case["task"], "where": case["where"], "config": cfg}
    if case["task"] == "batch":
        state["clouds"] = _batch_clouds(case, seed)
        state["first"] = np.cumsum([0] + [_max_tets(n) for n in _sizes(case)])
        rows = int(state["first"][-1])
        state["tets"], state["adjacency"] = (np.full((rows, 4), wt.INVALID, np.uint32) for _ in range(2))
        return state
    pts = _cloud(case["cloud"], case["n"], _gen(seed))
    state["points"] = pts.cpu().numpy() if case["where"] == "host" else pts
    if case["task"] == "verify":
        state["tets"], state["adjacency"] = (x.clone() for x in wt.delaunay_device(pts, cfg))
        return state
    rows = _max_tets(pts.shape[0])
    if case["where"] == "host":
        state["tets"], state["adjacency"] = (np.full((rows, 4), wt.INVALID, np.uint32) for _ in range(2))
    else:
        state["tets"], state["adjacency"] = (torch.full((rows, 4), -1, dtype=torch.int32, device="cuda")
                                             for _ in range(2))
    return state


def run(state):
    if state["task"] == "batch":
        results = wt.delaunay_batched(state["clouds"], state["config"])
        for cloud, r, o in zip(state["clouds"], results, state["first"]):
            t, a = wt.canonical(r.tets, r.adjacency, len(cloud))
            state["tets"][o:o + len(t)] = t
            state["adjacency"][o:o + len(a)] = a
        return {"tets": state["tets"], "adjacency": state["adjacency"]}
    pts = state["points"]
    if state["task"] == "verify":
        return wt.verify_device(pts, state["tets"], state["adjacency"])
    if state["where"] == "host":
        r = wt.delaunay(pts, state["config"])
        t, a = wt.canonical(r.tets, r.adjacency, len(pts))
        state["tets"][: len(t)] = t
        state["adjacency"][: len(a)] = a
        return {"tets": state["tets"], "adjacency": state["adjacency"], "failed": r.failed_verts}
    t, a = wt.delaunay_device(pts, state["config"])
    t, a = wt.canonical_device(t, a, pts.shape[0])
    state["tets"][: t.shape[0]] = t
    state["adjacency"][: a.shape[0]] = a
    return {"tets": state["tets"], "adjacency": state["adjacency"]}


# Tets per point of a finished triangulation (super vertices included), measured to a few percent.
_TETS = {"uniform": 6.7, "mixture": 6.7, "clustered": 6.7, "sphere": 5.05, "lattice": 6.1, "batch": 6.5}


def work(case):
    """Bytes: 12 per point read, 32 per tet (four ids, four links) written, or read by the check.  Operations: one
    insphere determinant (about 100) for each of the two faces a tet has to itself, which is what certifies the result."""
    if case["task"] == "batch":
        n = float(_sizes(case).sum())
    else:
        n = _points(case["cloud"], case["n"])
    tets = _TETS[case["cloud"]] * n
    return {"bytes": 12.0 * n + 32.0 * tets, "flops": 200.0 * tets}

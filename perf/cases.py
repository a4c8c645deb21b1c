"""What a program that uses gcdt_b200 has it do, as cases that can be timed.

  listed()             the named cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  what such a program holds before the call: inputs on the
                       device (or the host, for the server), the context
  run(state)           one pass through the public entry points -> its outputs
  work(case)           the bytes a pass cannot do without

The inputs are the distributions of the framework's own generators
(gcdt_b200.generate), made on the GPU because a 10M-point instance takes the
host generator seconds.  Every point set is distinct, in random order, the
polygon vertices last, as the generators leave it.

Outputs are integers throughout, so exact() has no value to give.
"""
import math

import numpy as np
import torch

import gcdt_b200 as g


def listed():
    return [
        # one small request on its own: an editor or a game that re-meshes a
        # shape after each change; latency and launches are all there is
        {"name": "solve_250", "kind": "solve", "dist": "uniform", "n": 250, "bits": 24, "polys": 1, "verts": 64},
        # the small end of the serving stream (requests from 1,000 points on)
        {"name": "solve_4k", "kind": "solve", "dist": "mixture", "n": 4001, "bits": 28, "polys": 1, "verts": 64},
        # the small plain-CDT configuration: 100k points in [1, 2^20), 512 segments
        {"name": "solve_small_100k", "kind": "solve", "dist": "uniform", "n": 100_512, "bits": 20, "polys": 8, "verts": 64},
        # the large end of the serving stream
        {"name": "solve_1m", "kind": "solve", "dist": "mixture", "n": 1_019_963, "bits": 28, "polys": 312, "verts": 64},
        # the headline: 10M points and 200k segments, terrain-like clusters
        {"name": "solve_scale_10m", "kind": "solve", "dist": "mixture", "n": 10_200_000, "bits": 30, "polys": 3125, "verts": 64},
        # plain Delaunay of uniform points over the whole box, no constraint
        {"name": "solve_uniform_9m", "kind": "solve", "dist": "uniform", "n": 9_000_000, "bits": 30, "polys": 0, "verts": 0},
        # gridded data, where every empty circle is a tie: 2048 x 2048 lattice, 20,000 unit segments
        {"name": "solve_lattice_2048", "kind": "solve", "dist": "lattice", "side": 2048, "segments": 20_000},
        # a handful of independent meshes per call (tiles, glyphs, parcels)
        {"name": "batch_256", "kind": "batch", "instances": 256, "smallest": 64, "largest": 65_536, "threads": 512, "stride": 16},
        # the batched configuration: 4,096 instances of 64 to 65,536 points
        {"name": "batch_4096", "kind": "batch", "instances": 4096, "smallest": 64, "largest": 65_536, "threads": 512, "stride": 16},
        # export of the scale mesh in the reference's renumbered layout
        {"name": "layout_10m", "kind": "layout", "dist": "mixture", "n": 10_200_000, "bits": 30, "polys": 3125, "verts": 64},
        # inside / outside of the scale mesh's polygons
        {"name": "regions_10m", "kind": "regions", "dist": "mixture", "n": 10_200_000, "bits": 30, "polys": 3125, "verts": 64},
        # a burst of requests at the server, submitted and fetched from host memory
        {"name": "serve_16", "kind": "serve", "requests": 16, "smallest": 1000, "largest": 300_000, "workers": 6},
    ]


def _log_uniform(rng, lo, hi):
    return int(math.floor(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_mesh(rng, lo, hi):
    dist = rng.choice(["uniform", "mixture", "mixture", "lattice"])
    if dist == "lattice":
        side = int(math.sqrt(_log_uniform(rng, max(lo, 1024), min(hi, 1 << 22))))
        return {"dist": dist, "side": side, "segments": rng.randrange(4, side * side // 200 + 5)}
    n = _log_uniform(rng, lo, hi)
    bits = rng.choice([20, 24, 28, 30]) if n <= 200_000 else rng.choice([28, 30])
    verts = rng.choice([16, 64, 64, 128]) if n >= 1000 else 16
    polys = rng.choice([0, n // 50 // verts, n // 50 // verts, n // 400 // verts + 1])
    return {"dist": dist, "n": n, "bits": bits, "polys": polys, "verts": verts if polys else 0}


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "batch", "layout", "regions"])
    if kind == "batch":
        inst = _log_uniform(rng, 3, 2048)
        return {"kind": kind, "instances": inst, "smallest": 64, "largest": _log_uniform(rng, 2000, 65_536),
                "threads": rng.choice([128, 256, 512]), "stride": rng.choice([16, 64])}
    lo, hi = (64, 8_000_000) if kind == "solve" else (1000, 8_000_000)
    return {"kind": kind, **_draw_mesh(rng, lo, hi)}


# ---------------------------------------------------------------- inputs

def _sizes(case):
    """Point counts of a batch's instances or a burst's requests: evenly
    spread over the logarithm, odd and even ones among them."""
    m = case["instances"] if case["kind"] == "batch" else case["requests"]
    lo, hi = case["smallest"], case["largest"]
    return [int(lo * (hi / lo) ** ((i + 0.5) / m)) for i in range(m)]


def _stars(cx, cy, r, verts, gen):
    """Star polygons around (cx, cy) (device tensors), `verts` vertices each
    (a host list): radii in [0.5 r, r], one angle in each equal sector.
    Returns vertices (sum, 2) int64 and, per vertex, its polygon's next one."""
    dev = cx.device
    nv = torch.tensor(verts, device=dev)
    poly = torch.repeat_interleave(torch.arange(len(verts), device=dev), nv)
    first = torch.cumsum(nv, 0) - nv
    k = torch.arange(len(poly), device=dev) - first[poly]
    u = torch.rand(2, len(poly), device=dev, dtype=torch.float64, generator=gen)
    ang = 2 * math.pi * (k + 0.1 + 0.8 * u[0]) / nv[poly]
    rad = r[poly] * (0.5 + 0.5 * u[1])
    xy = torch.stack([cx[poly] + rad * torch.cos(ang), cy[poly] + rad * torch.sin(ang)], 1).round().long()
    nxt = first[poly] + (k + 1) % nv[poly]
    return xy, nxt, poly


def _distinct(fixed, free, redraw):
    """Redraw entries of the key vector `free` until all of fixed + free differ."""
    while True:
        keys, at = torch.sort(torch.cat([fixed, free]), stable=True)
        again = at[1:][keys[1:] == keys[:-1]] - len(fixed)
        if len(again) == 0:
            return free
        free[again] = redraw(again)


def _mesh_input(case, seed, dev):
    """Points (n, 2) and segments (s, 2), int32 on the device."""
    if case["dist"] == "lattice":
        xy, cons = g.generate(g.GEN_LATTICE, seed, case["side"], case["segments"])
        return torch.from_numpy(xy).to(dev), torch.from_numpy(cons).to(dev)
    gen = torch.Generator(device=dev).manual_seed(seed)
    hi = (1 << case["bits"]) - 2
    polys, verts = case["polys"], case["verts"]
    if polys:
        side = math.ceil(math.sqrt(polys))
        cell = (1 << case["bits"]) / side
        at = torch.randperm(side * side, device=dev, generator=gen)[:polys]
        r = torch.full((polys,), math.floor(0.45 * cell), device=dev, dtype=torch.float64)
        star, nxt, _ = _stars((at % side + 0.5) * cell, (at // side + 0.5) * cell, r, [verts] * polys, gen)
    else:
        star = torch.empty((0, 2), device=dev, dtype=torch.int64)
        nxt = torch.empty(0, device=dev, dtype=torch.int64)
    m = case["n"] - polys * verts
    centres = torch.randint(1, hi + 1, (64, 2), device=dev, generator=gen)
    sigma = float(1 << (case["bits"] - 8))

    def points(k):
        xy = torch.randint(1, hi + 1, (k, 2), device=dev, generator=gen)
        if case["dist"] == "mixture":       # 90% in 64 Gaussians, 10% uniform
            which = torch.randint(0, 64, (k,), device=dev, generator=gen)
            near = centres[which] + (sigma * torch.randn(k, 2, device=dev, dtype=torch.float64, generator=gen)).round().long()
            xy = torch.where(torch.rand(k, 1, device=dev, generator=gen) < 0.9, near.clamp(1, hi), xy)
        return (xy[:, 0] << 32) | xy[:, 1]

    keys = _distinct((star[:, 0] << 32) | star[:, 1], points(m), lambda again: points(len(again)))
    xy = torch.cat([torch.stack([keys >> 32, keys & 0xffffffff], 1), star]).int().contiguous()
    segs = torch.stack([torch.arange(len(star), device=dev), nxt], 1) + m
    return xy, segs.int().contiguous()


def _batch_counts(case):
    """Per instance (in call order, large and small ones mixed): points besides
    the polygons', and the polygons' vertex counts."""
    r = np.random.RandomState(case["instances"] * 7 + case["largest"])
    out = []
    for n in r.permutation(_sizes(case)):
        verts = [int(r.randint(16, 257)) for _ in range(int(r.randint(1, 5)))] if n >= 1000 else [16]
        out.append((int(n), verts))
    return out


def _batch_input(case, seed, dev):
    """Concatenated instances: uniform points in [1, 2^24) and stars in
    distinct quadrants; segment indices are local to the instance."""
    gen = torch.Generator(device=dev).manual_seed(seed)
    counts = _batch_counts(case)
    free = torch.tensor([n for n, _ in counts], device=dev)
    corner = torch.tensor([sum(v) for _, v in counts], device=dev)
    npoly = torch.tensor([len(v) for _, v in counts], device=dev)
    ninst = len(counts)
    owner = torch.repeat_interleave(torch.arange(ninst, device=dev), npoly)      # of each polygon
    turn = torch.randint(0, 4, (ninst,), device=dev, generator=gen)[owner]
    quad = (torch.arange(len(owner), device=dev) - (torch.cumsum(npoly, 0) - npoly)[owner] + turn) % 4
    cell = float(1 << 23)
    r = torch.full((len(owner),), math.floor(0.45 * cell), device=dev, dtype=torch.float64)
    star, nxt, poly = _stars((quad % 2 + 0.5) * cell, (quad // 2 + 0.5) * cell, r, [v for _, vs in counts for v in vs], gen)
    star_inst = owner[poly]
    inst = torch.repeat_interleave(torch.arange(ninst, device=dev), free)

    def points(which):
        xy = torch.randint(1, 1 << 24, (len(which), 2), device=dev, generator=gen)
        return (inst[which] << 48) | (xy[:, 0] << 24) | xy[:, 1]

    keys = _distinct((star_inst << 48) | (star[:, 0] << 24) | star[:, 1],
                     points(torch.arange(len(inst), device=dev)), points)
    pts = free + corner
    po = torch.cumsum(pts, 0) - pts                      # first point of each instance
    xy = torch.empty((int(pts.sum()), 2), dtype=torch.int32, device=dev)
    at = po[inst] + torch.arange(len(inst), device=dev) - (torch.cumsum(free, 0) - free)[inst]
    xy[at] = torch.stack([(keys >> 24) & 0xffffff, keys & 0xffffff], 1).int()
    # the k-th polygon vertex of an instance is its point free + k
    before = (torch.cumsum(corner, 0) - corner)[star_inst]
    local = free[star_inst] + torch.arange(len(star), device=dev) - before
    xy[po[star_inst] + local] = star.int()
    cons = torch.stack([local, free[star_inst] + nxt - before], 1).int().contiguous()
    zero = np.zeros(1, np.int64)
    return (xy, cons, np.concatenate([zero, np.cumsum(pts.cpu().numpy())]),
            np.concatenate([zero, np.cumsum(corner.cpu().numpy())]))


# ---------------------------------------------------------------- the cases

def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    kind = case["kind"]
    if kind == "batch":
        xy, cons, po, so = _batch_input(case, seed, dev)
        bt = g.BatchTriangulator(len(po) - 1, int(po[-1]), int(so[-1]), device=dev.index)
        bt.set_config(case["threads"], case["stride"])
        return {"kind": kind, "bt": bt, "xy": xy, "cons": cons, "po": po, "so": so, "out": bt.alloc_outputs(po)}
    if kind == "serve":
        srv = g.Server(memory_budget_bytes=24 << 30, max_request_points=case["largest"] + 1, big_request_points=8000,
                       max_batch_points=400_000, big_workers=case["workers"], device=dev.index)
        reqs = []
        for i, n in enumerate(_sizes(case)):
            xy, cons = _mesh_input({"dist": "mixture", "n": n, "bits": 28, "polys": max(1, n // 3200), "verts": 16},
                                   seed * 1000 + i, dev)
            reqs.append((xy.cpu().numpy(), cons.cpu().numpy()))
        return {"kind": kind, "srv": srv, "reqs": reqs}
    xy, cons = _mesh_input(case, seed, dev)
    n, s = len(xy), len(cons)
    tri = g.Triangulator(max_points=n, max_segments=s, device=dev.index)
    T = 2 * n + 2
    out = (torch.empty((T, 3), dtype=torch.int32, device=dev), torch.empty((T, 3), dtype=torch.int32, device=dev),
           torch.empty((T,), dtype=torch.uint8, device=dev))
    if kind == "solve":
        return {"kind": kind, "tri": tri, "xy": xy, "cons": cons, "out": out}
    tri.triangulate(xy, cons, out=out)      # the mesh that the output-side calls start from
    tri.close()
    return {"kind": kind, "xy": xy, "mesh": out}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        return state["tri"].triangulate(state["xy"], state["cons"], out=state["out"])
    if kind == "batch":
        out, status, rc = state["bt"].triangulate_device(state["xy"], state["cons"], state["po"], state["so"],
                                                         out=state["out"])
        return out, status, rc
    if kind == "layout":
        return g.reference_layout(state["xy"], *state["mesh"])
    if kind == "regions":
        return g.classify_regions(state["mesh"][1], state["mesh"][2])
    srv = state["srv"]
    ids = [srv.submit(xy, cons) for xy, cons in state["reqs"]]
    got = []
    for rid, (xy, _) in zip(ids, state["reqs"]):
        srv.wait(rid)
        got.append(srv.fetch(rid, len(xy)))
        srv.release(rid)
    return got


def _mesh_size(case):
    if case["dist"] == "lattice":
        return case["side"] ** 2, case["segments"]
    return case["n"], case["polys"] * case["verts"]


def work(case):
    """Inputs read once and outputs written once; nothing here is a
    contraction, so there are no flops to count."""
    kind = case["kind"]
    if kind == "batch":
        counts = _batch_counts(case)
        s = sum(sum(v) for _, v in counts)
        n = s + sum(m for m, _ in counts)
        return {"bytes": 8 * n + 8 * s + 25 * (2 * n + 2 * len(counts)), "flops": 0}
    if kind == "serve":
        n, m = sum(_sizes(case)), case["requests"]
        s = sum(16 * max(1, k // 3200) for k in _sizes(case))
        return {"bytes": 8 * n + 8 * s + 25 * (2 * n + 2 * m), "flops": 0}
    n, s = _mesh_size(case)
    T = 2 * n + 2
    if kind == "layout":        # points and mesh in; points, labels and mesh out
        return {"bytes": 8 * n + 25 * T + 12 * (n + 4) + 25 * T, "flops": 0}
    if kind == "regions":       # adjacency and flags in, depth out
        return {"bytes": 17 * T, "flops": 0}
    return {"bytes": 8 * n + 8 * s + 25 * T, "flops": 0}


def exact(case, seed):
    """Every output is a whole number: nothing is rounded."""
    return None

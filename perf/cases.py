"""Workloads of the layout library as its users run them, one pass each.

A pass is one call sequence of a program that drives the library: a layout
step over positions in pinned host memory (``step_host``, what the
"forceEmbedder.step" action does per frame), a whole ``begin`` / ``run`` /
``positions`` layout, a GRIP refinement round with the positions going both
ways, the exact-repulsion judge of the learned walk, or a training call of the
far-field network. Steps run on: each pass continues the layout that the last
one left in the host buffer, as an iteration loop does.

The steps' outputs are the single-precision vertex buffer that a renderer
draws from.

``exact`` restates the passes in 64 bits with plain torch (a level-by-level
quadtree and a frontier walk, or all pairs), without the library.
"""
import math

import numpy as np
import torch

from grapher_b200 import ForceLayout, graphs
from grapher_b200 import _native as native
from grapher_b200.farfield import FarFieldModel
from grapher_b200.grip import GripRefiner, k_nearest

LINLOG = 1
EDGE = 10.0       # the embedder's default edge length
OVERLAP_C = 100.0  # the embedder's default overlap constant


def listed():
    return [
        # the smallest interactive layout: a 32 x 32 mesh, every launch counts
        dict(name="grid1k_step", kind="step", graph="grid", V=1024, model=0, theta=0.5,
             start="uniform", box=1.0),
        # an ordinary interactive graph at the embedder's default theta
        dict(name="ba5k_step", kind="step", graph="ba", V=4999, m=3, model=LINLOG, theta=1.0,
             gravity=1.0, start="settled", box=300.0),
        # a mid-sized layout well under way, tight opening threshold, odd size
        dict(name="ba65k_step", kind="step", graph="ba", V=65537, m=4, model=LINLOG, theta=0.5,
             gravity=1.0, start="settled", box=500.0),
        # a large scale-free graph from its random start, degree-sized radii kept apart
        dict(name="ba1m_overlap_step", kind="step", graph="ba", V=1048576, m=4, model=LINLOG,
             theta=0.8, gravity=1.0, overlap=True, start="uniform", box=1000.0),
        # the same size with the learned far field, hubs on the plain walk
        dict(name="ba1m_learned_step", kind="step", graph="ba", V=1048576, m=4, model=LINLOG,
             theta=1.225, gravity=1.0, learned=True, hub_targets=1024, start="settled",
             box=1000.0),
        # a skewed graph (hubs of thousands of neighbours) with the learned far field
        dict(name="rmat262k_learned_step", kind="step", graph="rmat", V=262144, m=8, model=LINLOG,
             theta=1.3, gravity=1.0, learned=True, hub_targets=4096, start="settled", box=700.0),
        # Barnes-Hut off: every pair, the exact mode
        dict(name="er65k_exact_step", kind="step", graph="er", V=65536, m=4, model=0, bh=False,
             start="disk", box=1.0),
        # many small uneven graphs laid out together
        dict(name="batch512_step", kind="step", graph="batch", count=512, model=0, theta=0.7,
             start="uniform", box=0.0),
        # a whole layout in the double-precision mode, stopped by its round limit
        dict(name="ba20k_fp64_run", kind="run", graph="ba", V=20000, m=4, model=LINLOG, theta=0.8,
             gravity=1.0, fp64=True, rounds=5, start="uniform", box=150.0),
        # GRIP's finest layer: every vertex, edges and k nearest
        dict(name="grip100k_fine_round", kind="grip", V=100000, m=3, k=128, layer=0, active=100000),
        # the learned workflow beside the step: exact forces of the judge's sampled vertices
        dict(name="judge_131k", kind="judge", graph="ba", V=131072, m=4, model=LINLOG,
             targets=4096, start="settled", box=500.0),
        # ... and an epoch of training on harvested pairs
        dict(name="mlp_train", kind="train", n=100000, epochs=1, batch=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["step", "step", "step", "overlap", "learned", "exact", "batch", "run",
                       "grip", "grip", "judge", "train"])
    model = rng.choice([0, LINLOG])
    start = rng.choice(["uniform", "settled"])
    if what in ("step", "overlap", "learned"):
        # FR on bounded degrees, LinLog (with or without radii) on any
        graph = rng.choice(["er", "grid"] if model != LINLOG else ["ba", "ba", "er", "grid"])
        c = dict(kind="step", graph=graph, V=_log_int(rng, 300, 900000), m=rng.randint(2, 5),
                 model=model, theta=round(rng.uniform(0.5, 1.2), 3),
                 gravity=rng.choice([0.0, 1.0]), start=start)
        if what == "overlap":
            c.update(model=LINLOG, overlap=True)
        if what == "learned":
            c.update(model=LINLOG, gravity=1.0, V=_log_int(rng, 20000, 900000), learned=True,
                     hub_targets=rng.choice([0, 256, 1024]), theta=round(rng.uniform(1.0, 1.3), 3))
        c.update(box=0.5 * EDGE * math.sqrt(c["V"]) * rng.uniform(0.2, 1.0))
        return c
    if what == "exact":
        return dict(kind="step", graph="er", V=_log_int(rng, 500, 60000), m=4, model=model,
                    bh=False, overlap=model == LINLOG and rng.random() < 0.5, start="disk",
                    box=rng.choice([1.0, 300.0]))
    if what == "batch":
        return dict(kind="step", graph="batch", count=_log_int(rng, 16, 500), model=0,
                    theta=round(rng.uniform(0.5, 1.0), 3), start="uniform", box=0.0)
    if what == "run":
        V = _log_int(rng, 500, 20000)
        return dict(kind="run", graph="ba", V=V, m=rng.randint(2, 5), model=model, gravity=1.0,
                    theta=round(rng.uniform(0.6, 1.2), 3), fp64=True, rounds=rng.randint(2, 5),
                    start="uniform", box=math.sqrt(V))
    if what == "grip":  # the finest layer, or a coarse one: springs to the k nearest active
        V = _log_int(rng, 2000, 100000)
        if rng.random() < 0.5:
            return dict(kind="grip", V=V, m=rng.randint(2, 4), k=rng.randint(8, 128), layer=0,
                        active=V)
        return dict(kind="grip", V=V, m=rng.randint(2, 4), k=rng.randint(8, 64),
                    layer=rng.randint(1, 5), active=max(100, int(V * rng.uniform(0.02, 0.5))))
    if what == "judge":
        return dict(kind="judge", graph="ba", V=_log_int(rng, 10000, 250000), m=4, model=LINLOG,
                    targets=_log_int(rng, 500, 4096), start=start, box=500.0)
    return dict(kind="train", n=_log_int(rng, 5000, 100000), epochs=1,
                batch=rng.choice([1024, 4096]))


# ------------------------------------------------------------------- inputs
def _graph(case, seed):
    """(row, col, graph offsets or None, number of vertices)"""
    kind = case["graph"]
    if kind == "batch":
        sizes = np.random.default_rng([case["count"], 0])  # the case's own, of any seed
        rng = np.random.default_rng([seed, 1])
        parts = []
        for g in range(case["count"]):
            V = int(round(math.exp(sizes.uniform(math.log(32), math.log(8192)))))
            shape = int(sizes.integers(3))
            s = int(rng.integers(1 << 30))
            if shape == 0:
                a, b = graphs.erdos_renyi(V, int(round(V * rng.uniform(3.0, 6.0) / 2)), s)
            elif shape == 1:
                a, b = graphs.random_connected(V, 0.0, s)
            else:
                side = max(1, int(round(math.sqrt(V))))
                V = side * side
                a, b = graphs.grid(side, side)
            parts.append((V, a, b))
        row, col, off = graphs.batch(parts)
        return row, col, off, int(off[-1])
    V = case["V"]
    if kind == "grid":
        rows = max(1, int(math.sqrt(V)))
        V = rows * (V // rows)
        a, b = graphs.grid(rows, V // rows)
    elif kind == "ba":
        a, b = graphs.barabasi_albert(V, case["m"], seed)
    elif kind == "rmat":
        scale = int(round(math.log2(V)))
        V = 1 << scale
        a, b = graphs.rmat(scale, case["m"] * V, seed=seed)
    else:
        a, b = graphs.erdos_renyi(V, case["m"] * V, seed)
    row, col = graphs.to_csr(V, a, b)
    return row, col, None, V


def _start(case, seed, V, off):
    """Interleaved float64 positions: uniform in the box (a layout's first
    frame), a settled layout (a dense core, clumps around it) or the disk."""
    rng = np.random.default_rng([seed, 2])
    if off is not None:  # each graph in its own default box
        sizes = np.diff(off).astype(np.int64)
        box = np.repeat(0.5 * EDGE * np.sqrt(sizes), sizes)[:, None]
        return (rng.uniform(-1.0, 1.0, (V, 2)) * box).reshape(-1)
    box = case["box"]
    if case["start"] == "disk":
        r, t = box * np.sqrt(rng.random(V)), 2.0 * np.pi * rng.random(V)
        return np.stack([r * np.cos(t), r * np.sin(t)], 1).reshape(-1)
    if case["start"] == "uniform":
        return rng.uniform(-box, box, 2 * V)
    centre = rng.normal(0.0, 0.45 * box, (max(4, V // 2000), 2))
    which = rng.integers(0, len(centre), V)
    clump = centre[which] + rng.normal(0.0, 0.04 * box, (V, 2))
    core = rng.normal(0.0, 0.3 * box, (V, 2))
    return np.where(rng.random((V, 1)) < 0.35, clump, core).reshape(-1)


def _weights(seed):
    """Random weights of the far-field network in its master layout
    (w1t[64][16], b1, w2t[64][64], b2, w3t[8][64], b3[8]), small outputs."""
    rng = np.random.default_rng([seed, 3])
    w1 = np.zeros((64, 16))
    w1[:, :10] = rng.normal(0.0, math.sqrt(2.0 / 10), (64, 10))
    w2 = rng.normal(0.0, math.sqrt(2.0 / 64), (64, 64))
    w3 = np.zeros((8, 64))
    w3[:2] = rng.normal(0.0, 0.02, (2, 64))
    zeros = np.zeros(64)
    return np.concatenate([w1.ravel(), zeros, w2.ravel(), zeros, w3.ravel(),
                           np.zeros(8)]).astype(np.float32)


def _layout(case, seed):
    row, col, off, V = _graph(case, seed)
    lay = ForceLayout(row, col, model=case["model"], graph_offsets=off)
    net = None
    if case.get("learned"):
        net = FarFieldModel(seed=1)
        net.set_weights(_weights(seed))
        net.attach(lay)
    over = case.get("overlap", False)
    lay.set_params(theta=case.get("theta", 1.0), gravityK=case.get("gravity", 0.0),
                   barnesHutEnabled=int(case.get("bh", True)),
                   precision=native.FP64 if case.get("fp64") else native.FP32,
                   preventOverlap=int(over), radiusBase=1.0 if over else 0.0,
                   radiusPerDegree=0.5 if over else 0.0)
    if net is not None:
        lay.set_params(farField=1, farCellGroups=1, farHubTargets=case["hub_targets"])
    x0 = _start(case, seed, V, off)
    return dict(layout=lay, net=net, x0=x0, V=V)


def _pinned(values):
    t = torch.empty(len(values), dtype=torch.float64, pin_memory=torch.cuda.is_available())
    t.numpy()[:] = values
    return t


def _grip(case, seed):
    """The graph's CSR, the layer's active vertices in a random filtration
    order, their k nearest among them, and positions."""
    a, b = graphs.barabasi_albert(case["V"], case["m"], seed)
    row, col = graphs.to_csr(case["V"], a, b)
    rng = np.random.default_rng([seed, 4])
    V, n = case["V"], case["active"]
    act = rng.permutation(V)[:n].astype(np.uint32)
    visible = np.zeros(V, np.uint8)
    visible[act] = 1
    off, kv, kd = k_nearest(row, col, act, case["k"], visible=None if n == V else visible)
    return row, col, act, off, kv, kd, rng.uniform(-1000.0, 1000.0, 2 * V)


def _samples(case, seed):
    """Feature / target / weight triples of the far field's ranges: h/d
    powers, rotated second moments, offsets, log2 counts; a smooth target."""
    rng = np.random.default_rng([seed, 5])
    n = case["n"]
    s = rng.uniform(0.05, 0.6, n)
    X = np.stack([s, rng.normal(0, 0.1, n) * s * s, rng.normal(0, 0.1, n) * s * s,
                  rng.uniform(0.1, 0.6, n) * s * s, rng.uniform(0, 0.1, n),
                  rng.uniform(-1, 1, n), rng.uniform(-1, 1, n), rng.uniform(1, 16, n),
                  s * s, s ** 3], 1).astype(np.float32)
    T = np.stack([X[:, 1] / (s * s) + 0.2 * s, X[:, 2] / (s * s)], 1)
    T = (T + rng.normal(0, 0.02, T.shape)).astype(np.float32)
    W = rng.exponential(1.0, n).astype(np.float32)
    return X, T, W


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "run"):
        s = _layout(case, seed)
        if kind == "step":
            s["pinned"] = _pinned(s["x0"])
            s["frame"] = torch.empty(len(s["x0"]), dtype=torch.float32)
            s["layout"].begin(0, positions=s["x0"])
    elif kind == "judge":
        s = _layout(case, seed)
        # a layout in progress, at the positions it is judged on
        s["layout"].begin(0, positions=s["x0"])
        s["layout"].step()
        s["layout"].set_positions(s["x0"])
        s["targets"] = np.sort(np.random.default_rng([seed, 6]).permutation(s["V"])
                               [:case["targets"]]).astype(np.uint32)
    elif kind == "grip":
        row, col, act, off, kv, kd, x0 = _grip(case, seed)
        g = GripRefiner(row, col)
        g.set_layer(case["layer"], act, off, kv, kd)
        s = dict(grip=g, xy=x0)
    else:
        X, T, W = _samples(case, seed)
        net = FarFieldModel(seed=1)
        s = dict(net=net, w0=_weights(seed), X=X, T=T, W=W)
    s["case"] = case
    return s


# --------------------------------------------------------------------- pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        # one iteration end to end over the program's host positions, then
        # its float vertex buffer and the step's stats (both as precise as
        # the single-precision forces behind them)
        s["layout"].step_host(s["pinned"].numpy())
        s["frame"].copy_(s["pinned"])
        stats = np.frombuffer(s["layout"].last_stats, np.float64).reshape(-1, 5)
        return dict(positions=s["frame"], stats=stats.astype(np.float32))
    if kind == "run":
        lay = s["layout"]
        lay.begin(0, positions=s["x0"])
        rounds = lay.run(case["rounds"], 1e-6)
        return dict(positions=lay.positions(), rounds=rounds)
    if kind == "judge":
        return dict(force=s["layout"].exact_repulsion(s["targets"]))
    if kind == "grip":
        g = s["grip"]
        g.set_positions(s["xy"])
        stats = g.refine_round()
        s["xy"] = g.positions()
        return dict(positions=s["xy"], stats=stats)
    net = s["net"]
    net.set_weights(s["w0"])
    loss = net.train(s["X"], s["T"], s["W"], epochs=case["epochs"], batch=case["batch"])
    return dict(loss=loss, weights=net.weights())


# --------------------------------------------------------------------- work
def _batch_vertices(case):
    return case["count"] * (8192 - 32) / math.log(8192 / 32)


def work(case):
    kind = case["kind"]
    if kind == "train":
        n = case["n"] * case["epochs"]
        return {"bytes": n * 52, "flops": n * 3 * 2 * (10 * 64 + 64 * 64 + 64 * 2)}
    if kind == "grip":
        n, k = case["active"], case["k"]
        edges = 2 * case["m"] * case["V"] if case["layer"] == 0 else 0
        # lists (id, distance) and adjacency once, positions and the
        # vertices' heat, displacement, cosine in and out
        return {"bytes": n * k * 8 + edges * 4 + case["V"] * 32 + n * 80,
                "flops": (n * k + edges) * 14}
    if kind == "judge":
        return {"bytes": case["V"] * 24 + case["targets"] * 20,
                "flops": 20.0 * case["V"] * case["targets"]}
    if case["graph"] == "batch":
        V, degree = _batch_vertices(case), 3.5
        n = V / case["count"]
    else:
        V, degree = case["V"], 2 * case.get("m", 2)
        n = V
    if case.get("bh", True):
        # terms per vertex of a Barnes-Hut walk on a 2-D quadtree
        terms = min(n, 8.0 / case["theta"] ** 2 * math.log(max(n, 4), 4))
    else:
        terms = n
    steps = case.get("rounds", 1)
    # positions and the previous force in, positions, force and the speed
    # rule's per-vertex sums out, structure (adjacency, mass, degree) in
    return {"bytes": steps * V * (16 + 16 + 16 + 16 + 16 + 16 + 4 * degree),
            "flops": steps * V * (20.0 * terms + 12.0 * degree + 40.0)}


# ------------------------------------------------------- the same in 64 bits
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _tree(pos, gid, G):
    """Quadtree of leaf capacity 1 per graph, level by level. Returns node
    arrays (half size, mass slots to fill, child ranges) and each point's
    path of nodes, as (level node ids of the points still descending)."""
    dev = pos.device
    big = torch.full((G, 2), math.inf, dtype=pos.dtype, device=dev)
    lo = big.scatter_reduce(0, gid[:, None].expand(-1, 2), pos, "amin")
    hi = (-big).scatter_reduce(0, gid[:, None].expand(-1, 2), pos, "amax")
    span = (hi - lo).amax(1)
    half = torch.where(span > 0, span / 2, torch.ones_like(span))
    centre = (lo + hi) / 2
    node, point = gid.clone(), torch.arange(len(pos), device=dev)
    c, h = centre[gid], half[gid]
    halves, kids0, kidsN, members = [half], [], [], [(point, node)]
    base, count = 0, G
    while True:
        per = torch.bincount(node - base, minlength=count)
        deep = (per[node - base] > 1) & (h > 1e-9)
        start = torch.full((count,), -1, dtype=torch.int64, device=dev)
        number = torch.zeros(count, dtype=torch.int64, device=dev)
        kids0.append(start)
        kidsN.append(number)
        if not bool(deep.any()):
            break
        point, node, c, h = point[deep], node[deep], c[deep], h[deep]
        p = pos[point]
        east, north = p[:, 0] >= c[:, 0], p[:, 1] >= c[:, 1]
        h = h / 2
        c = torch.stack([torch.where(east, c[:, 0] + h, c[:, 0] - h),
                         torch.where(north, c[:, 1] + h, c[:, 1] - h)], 1)
        key = (node - base) * 4 + torch.where(north, 0, 2) + torch.where(east, 1, 0)
        uniq, inverse = torch.unique(key, return_inverse=True)
        nxt = base + count
        parent = uniq // 4
        number.scatter_add_(0, parent, torch.ones_like(parent))
        first = torch.searchsorted(parent, torch.arange(count, device=dev))
        has = number > 0
        start[has] = nxt + first[has]
        node = nxt + inverse
        hn = torch.zeros(len(uniq), dtype=pos.dtype, device=dev)
        hn[inverse] = h
        halves.append(hn)
        members.append((point, node))
        base, count = nxt, len(uniq)
    return torch.cat(halves), torch.cat(kids0), torch.cat(kidsN), members


def _term(model, d, mv, mo, radii):
    dist = d.square().sum(1).sqrt()
    gap = dist - radii
    num = mv * mo if model == LINLOG else torch.full_like(mo, EDGE * EDGE)
    mag = torch.where(gap > 0, num / gap, num * OVERLAP_C)
    if model != LINLOG:
        mag = mag * torch.floor(mo)
    return -(mag / dist)[:, None] * d


def _walk(case, pos, mass, radius, gid, G):
    """Barnes-Hut repulsion with the reference's per-target decisions."""
    half, kids0, kidsN, members = _tree(pos, gid, G)
    n = len(half)
    dev = pos.device
    M = torch.zeros(n, dtype=pos.dtype, device=dev)
    S = torch.zeros((n, 2), dtype=pos.dtype, device=dev)
    leaf = torch.zeros(len(pos), dtype=torch.int64, device=dev)
    for point, node in members:
        M.index_add_(0, node, mass[point])
        S.index_add_(0, node, mass[point][:, None] * pos[point])
        leaf[point] = node
    com = S / M[:, None]
    order = torch.argsort(leaf, stable=True)
    held = torch.bincount(leaf, minlength=n)
    first = torch.cumsum(held, 0) - held
    out = torch.zeros_like(pos)
    model, theta = case["model"], case["theta"]

    def spread(t, start, number):
        t = torch.repeat_interleave(t, number)
        at = torch.repeat_interleave(start - (torch.cumsum(number, 0) - number), number)
        return t, at + torch.arange(len(t), device=dev)

    for v0 in range(0, len(pos), 1 << 16):
        t = torch.arange(v0, min(v0 + (1 << 16), len(pos)), device=dev)
        node = gid[t]
        while len(t):
            is_leaf = kidsN[node] == 0
            tl, at = spread(t[is_leaf], first[node[is_leaf]], held[node[is_leaf]])
            u = order[at]
            tl, u = tl[u != tl], u[u != tl]
            out.index_add_(0, tl, _term(model, pos[u] - pos[tl], mass[tl], mass[u],
                                        radius[tl] + radius[u]))
            t, node = t[~is_leaf], node[~is_leaf]
            d = com[node] - pos[t]
            near = (2.0 * half[node]) / d.square().sum(1).sqrt() < theta
            out.index_add_(0, t[near], _term(model, d[near], mass[t[near]], M[node[near]],
                                             radius[t[near]]))
            t, node = t[~near], node[~near]
            t, node = spread(t, kids0[node], kidsN[node])
    return out


def _pairs(case, pos, mass, radius, targets):
    out = torch.zeros((len(targets), 2), dtype=pos.dtype, device=pos.device)
    step = max(1, (1 << 24) // len(pos))
    num_fr = EDGE * EDGE
    for i in range(0, len(targets), step):
        t = targets[i:i + step]
        d = pos[None, :, :] - pos[t][:, None, :]
        dist = d.square().sum(2).sqrt()
        num = mass[t][:, None] * mass[None, :] if case["model"] == LINLOG else num_fr
        gap = dist - (radius[t][:, None] + radius[None, :])
        mag = torch.where(gap > 0, num / gap, num * torch.full_like(gap, OVERLAP_C))
        f = torch.where(dist > 0, mag / dist, 0.0)
        out[i:i + step] = -(f[:, :, None] * d).sum(1)
    return out


class _Exact:
    """A layout's state in 64 bits and its step."""

    def __init__(self, case, seed):
        row, col, off, V = _graph(case, seed)
        dev = _device()
        self.case = case
        self.off = np.array([0, V], np.int64) if off is None else off.astype(np.int64)
        sizes = torch.from_numpy(np.diff(self.off)).to(dev)
        self.G, self.n, self.sizes = len(sizes), sizes.double(), sizes
        self.gid = torch.repeat_interleave(torch.arange(self.G, device=dev), sizes)
        self.pos = torch.from_numpy(_start(case, seed, V, off)).to(dev).reshape(-1, 2)
        deg = torch.from_numpy(np.diff(row).astype(np.int64)).to(dev)
        self.deg = deg.double()
        self.src = torch.repeat_interleave(torch.arange(V, device=dev), deg)
        self.dst = torch.from_numpy(col.astype(np.int64)).to(dev)
        self.mass = 1.0 + self.deg if case["model"] == LINLOG else torch.ones_like(self.deg)
        over = case.get("overlap", False)
        self.radius = (1.0 + 0.5 * self.deg.sqrt()) if over else torch.zeros_like(self.deg)
        self.old = torch.zeros_like(self.pos)
        self.speed = torch.ones_like(self.n)
        self.eff = torch.ones_like(self.n)

    def per_graph(self, x):
        # in one order for every x: the speed rule compares sums whose terms
        # are exact multiples of one another on a layout's first step
        return torch.segment_reduce(x, "sum", lengths=self.sizes)

    def step(self):
        case, pos = self.case, self.pos
        d = pos[self.dst] - pos[self.src]
        dist = d.square().sum(1).sqrt()
        s = torch.log(1.0 + dist) / dist if case["model"] == LINLOG else dist / EDGE
        s = torch.where(dist < 1e-9, 0.0, s)
        att = torch.zeros_like(pos).index_add_(0, self.src, s[:, None] * d)
        if case.get("bh", True):
            rep = _walk(case, pos, self.mass, self.radius, self.gid, self.G)
        else:
            rep = _pairs(case, pos, self.mass, self.radius,
                         torch.arange(len(pos), device=pos.device))
        f = att + rep
        norm = lambda x: x.square().sum(1).sqrt()  # noqa: E731
        swing = self.mass * norm(f - self.old)
        traction = 0.5 * self.mass * norm(f + self.old)
        gravity = case.get("gravity", 0.0)
        r = norm(pos)[:, None]
        g = gravity * (self.deg + 1.0)[:, None] / r * pos
        disp = f - torch.where(r < 1e-9, 0.0, g)
        self.old = f
        # ForceAtlas2's global speed
        sw, tr, n = self.per_graph(swing), self.per_graph(traction), self.n
        best = 0.05 * n.sqrt()
        jt = torch.maximum(best.sqrt(), torch.clamp(best * tr / (n * n), max=10.0))
        eff, speed = self.eff, self.speed
        rough = sw / tr > 2.0
        eff = torch.where(rough & (eff > 0.05), eff * 0.5, eff)
        jt = torch.where(rough, torch.clamp(jt, min=1.0), jt)
        target = torch.where(sw > 1e-7, jt * eff * tr / sw, speed)
        wild = sw > jt * tr
        eff = torch.where(wild, torch.where(eff > 0.05, eff * 0.7, eff),
                          torch.where(speed < 1000.0, eff * 1.3, eff))
        eff = torch.clamp(eff, 0.05, 1.0)
        moved = speed + torch.minimum(target - speed, 0.5 * speed)
        still = tr < 1e-7
        self.eff = torch.where(still, self.eff, eff)
        self.speed = torch.where(still, self.speed, moved)
        v = self.speed[self.gid]
        o = disp * (v / (1.0 + (v * swing).sqrt()))[:, None]
        self.pos = pos + o
        top = torch.zeros_like(n).scatter_reduce(0, self.gid, norm(o), "amax")
        return torch.stack([top, self.speed, self.per_graph(norm(att)) / n,
                            self.per_graph(norm(rep)) / n,
                            gravity * self.per_graph(self.deg + 1.0) / n], 1)


def _exact_grip(case, seed):
    row, col, act, off, kv, kd, x0 = _grip(case, seed)
    dev = _device()
    pos = torch.from_numpy(x0).to(dev).reshape(-1, 2)
    on = lambda x: torch.from_numpy(np.asarray(x).astype(np.int64)).to(dev)  # noqa: E731
    a = on(act)
    t = torch.repeat_interleave(a, on(np.diff(off)))
    near, dist = on(kv), on(kd).double()
    f = torch.zeros_like(pos)
    if case["layer"] > 0:
        length = dist * EDGE
        d = pos[near] - pos[t]
        s = torch.where(length < 1e-9, 0.0, d.square().sum(1).sqrt() / length - 1.0)
        f.index_add_(0, t, s[:, None] * d)
    else:
        src = torch.repeat_interleave(torch.arange(len(pos), device=dev), on(np.diff(row)))
        d = pos[on(col)] - pos[src]
        f.index_add_(0, src, d.square().sum(1)[:, None] / (EDGE * EDGE) * d)
        d = pos[t] - pos[near]
        d2 = d.square().sum(1)
        f.index_add_(0, t, torch.where(d2 < 1e-18, 0.0, 0.05 * EDGE * EDGE / d2)[:, None] * d)
    p, f = pos[a], f[a]
    force = f.square().sum(1).sqrt()
    heat = EDGE / 6.0  # the first round of a layer
    step = torch.where((force > 1e-7)[:, None], heat / force[:, None] * f, f)
    step = step - step.mean(0)
    r = p - p.mean(0)
    inertia = r.square().sum()
    if len(a) >= 3 and float(inertia) >= 1e-7:
        w = (r[:, 0] * step[:, 1] - r[:, 1] * step[:, 0]).sum() / inertia
        step = step - torch.stack([-w * r[:, 1], w * r[:, 0]], 1)
    pos[a] = p + step
    size = step.square().sum(1).sqrt()
    stats = np.array([float(size.max()), float(size.mean()), float(force.mean()), heat])
    return dict(positions=pos.reshape(-1).cpu().numpy(), stats=stats)


def exact(case, seed):
    kind = case["kind"]
    if kind == "train" or case.get("learned"):
        return None  # 16-bit networks by definition: no 64-bit value of these outputs
    if case.get("overlap"):
        # a pair's force grows without bound as its gap closes: among many
        # pairs, some gap is below single precision's resolution of it
        return None
    if kind == "grip":
        return _exact_grip(case, seed)
    e = _Exact(case, seed)
    if kind == "judge":
        t = np.sort(np.random.default_rng([seed, 6]).permutation(len(e.pos))[:case["targets"]])
        return dict(force=_pairs(case, e.pos, e.mass, e.radius,
                                 torch.from_numpy(t).to(e.pos.device)).cpu().numpy())
    if kind == "run":
        for _ in range(case["rounds"]):
            e.step()
        return dict(positions=e.pos.reshape(-1).cpu().numpy(), rounds=None)
    stats = e.step()
    return dict(positions=e.pos.reshape(-1).cpu().numpy(), stats=stats.cpu().numpy())

"""Performance cases of the framework: what a program that uses it has it do,
through the public Python API (and, for the entry point without a context, the
C ABI), from a small game level to the largest maze batch.

A case is a dict of plain values:

  kind     "frames"   retarget a share of the agents, then step (GMAPF)
           "search"   a batch of path queries on device buffers (search_batch_device)
           "noalloc"  the same through gmapf_search_batch_noalloc
           "scenes"   several worlds stepped as one (SceneBatch)
           "serve"    retargets served as they arrive, then the frame that installs them
  map      "maze" (size = cells per side, 4000 x 4000, walls 4 wide) or
           "rects" (size = rectangles with sides 10..60 in a square)
  agents   agents, or queries
  T, C     threads per agent and queue capacity (the Config's two search parameters)
  retarget share of the agents that get a new target in each pass
  steps    frames in one pass
  mode     0 batched (a CUDA graph per frame), 1 plain (one launch per chunk of requests)
  smooth   path smoothing (0 off, 1 funnel corners, 2 corners one radius off the walls)
"""
from __future__ import annotations

import math

import numpy as np
import torch

from gmapf_b200 import GMAPF, SceneBatch, make_config
from gmapf_b200 import _lib
from gmapf_b200.api import NODE_DTYPE
from gmapf_b200.scenarios import maze_walls, random_rects

MAZE_SIDE, MAZE_WALL = 4000.0, 4.0
DT = 1.0 / 60.0
STATS = ("requests", "found", "expansions", "rounds", "deg_sum", "claims", "path_nodes", "moving", "neighbours")


def _case(kind, map, size, agents, T, C, retarget=1.0, steps=1, mode=0, smooth=0, scenes=1):
    return dict(kind=kind, map=map, size=size, agents=agents, T=T, C=C, retarget=retarget, steps=steps, mode=mode,
                smooth=smooth, scenes=scenes)


def listed():
    named = {
        # a small level in which every agent is sent somewhere else in one frame: launch and host latency
        "frame_256": _case("frames", "rects", 4, 256, 4, 16),
        # the usual frame of a mid-size world: everybody walks, nobody searches
        "walk_2k": _case("frames", "rects", 200, 2048, 8, 32, retarget=0.0),
        # the frame of that world in which everybody is retargeted, and the next one
        "retarget_2k": _case("frames", "rects", 200, 2048, 8, 32, steps=2),
        # the same with steering through funnel corners: paths start in the second frame
        "smooth_2k": _case("frames", "rects", 200, 2048, 8, 32, steps=2, smooth=1),
        # a large crowd walking long corridors (long path rows, collisions)
        "walk_16k_maze": _case("frames", "maze", 64, 16384, 32, 16, retarget=0.0),
        # the full-retarget frame of the 64 x 64 maze at the shape the autotuner picks
        "frame_16k_maze64": _case("frames", "maze", 64, 16384, 32, 16),
        # the largest: the full-retarget frame of the ~100k-triangle maze at the tuned shape
        "frame_16k_maze160": _case("frames", "maze", 160, 16384, 32, 16),
        # the same maze as a batch of queries at the Config's own shape (odd count)
        "search_2k_maze160": _case("search", "maze", 160, 2047, 8, 32),
        # a few long queries at once: the latency of one search
        "search_few_maze64": _case("search", "maze", 64, 37, 32, 16),
        # the entry point for callers that may not allocate
        "noalloc_2k_maze64": _case("noalloc", "maze", 64, 2048, 8, 32),
        # many small scenes stepped as one, a few retargets per frame
        "scenes_64": _case("scenes", "rects", 60, 24000, 8, 32, retarget=0.02, scenes=64),
        # a burst of retargets through the serving form and the frame that installs them
        "serve_4k": _case("serve", "rects", 200, 4096, 8, 32),
    }
    return [dict(c, name=k) for k, c in named.items()]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frames"] * 6 + ["search"] * 3 + ["noalloc", "scenes", "serve"])
    if kind == "scenes":
        return _case(kind, "rects", _log(rng, 10, 80), _log(rng, 2000, 30000), rng.choice([4, 8, 16]),
                     rng.choice([16, 32]), retarget=rng.choice([0.0, 0.02, 0.2]), scenes=rng.randint(2, 64))
    if kind == "serve":
        return _case(kind, "rects", _log(rng, 20, 200), _log(rng, 256, 8192), rng.choice([4, 8, 32]),
                     rng.choice([16, 32]))
    maze = rng.random() < 0.5
    size = _log(rng, 12, 128) if maze else _log(rng, 4, 200)
    T = rng.choice([8, 16, 32, 32] if maze else [2, 4, 8, 16, 32])
    C = rng.choice([16, 32, 64])
    if kind != "frames":
        if kind == "noalloc" and maze:
            size = min(size, 64)
        return _case(kind, "maze" if maze else "rects", size, _log(rng, 16, 2048 if maze else 8192), T, C)
    retarget = rng.choice([0.0, 1.0, 1.0, round(rng.uniform(0.02, 0.5), 3)])
    mode, smooth = rng.choice([0, 0, 0, 1]), rng.choice([0, 0, 0, 1, 2])
    most = 1024 if maze and (mode or smooth) else 8192
    return _case(kind, "maze" if maze else "rects", size, _log(rng, 100, most), T, C, retarget=retarget,
                 steps=rng.choice([1, 1, 2, 3]), mode=mode, smooth=smooth)


# ---- navmeshes (gmapf_node records for FillMapManually) ---------------------

def _pack(vert, tri):
    """vert (v, 2), tri (n, 3) -> NODE_DTYPE records with packed neighbours."""
    n = len(tri)
    nodes = np.zeros(n, NODE_DTYPE)
    for k, f in enumerate(("P1", "P2", "P3")):
        nodes[f] = vert[tri[:, k]]
    a = np.concatenate([tri[:, 0], tri[:, 1], tri[:, 2]]).astype(np.int64)
    b = np.concatenate([tri[:, 1], tri[:, 2], tri[:, 0]]).astype(np.int64)
    key = np.minimum(a, b) * len(vert) + np.maximum(a, b)
    order = np.argsort(key, kind="stable")
    same = key[order][1:] == key[order][:-1]
    i, j = order[:-1][same], order[1:][same]
    nb = np.full((3 * n,), -1, np.int64)
    nb[i], nb[j] = j % n, i % n
    nb = nb.reshape(3, n).T
    idx = np.argsort(nb < 0, axis=1, kind="stable")  # existing neighbours first, in edge order
    nodes["NeibsIdx"] = np.take_along_axis(nb, idx, 1)
    return nodes


def _maze(cells, seed=3):
    """The randomized-DFS maze of scenarios.maze_walls: every free cell between the walls' coordinates as two
    triangles."""
    t, step = MAZE_WALL / 2, MAZE_SIDE / cells
    lines = np.concatenate([[0.0, t], *[[k * step - t, k * step + t] for k in range(1, cells)],
                            [MAZE_SIDE - t, MAZE_SIDE]])
    free = np.ones((len(lines) - 1, len(lines) - 1), bool)  # [y, x]
    at = lambda v: int(np.argmin(np.abs(lines - v)))  # noqa: E731
    for r in maze_walls(cells, MAZE_SIDE, MAZE_WALL, seed):
        free[at(r[:, 1].min()):at(r[:, 1].max()), at(r[:, 0].min()):at(r[:, 0].max())] = False
    m = len(lines)
    vert = np.stack([np.tile(lines, m), np.repeat(lines, m)], 1).astype(np.float32)
    y, x = np.nonzero(free)
    a, b, c, d = y * m + x, y * m + x + 1, (y + 1) * m + x + 1, (y + 1) * m + x
    flip = np.random.default_rng(seed).random(len(y)) < 0.5
    one = np.where(flip[:, None], np.stack([a, b, d], 1), np.stack([a, b, c], 1))
    two = np.where(flip[:, None], np.stack([b, c, d], 1), np.stack([a, c, d], 1))
    return _pack(vert, np.stack([one, two], 1).reshape(-1, 3))


def _rects(count, seed):
    """Delaunay triangles (incremental, Bowyer 1981 / Watson 1981) of a square with `count` rectangles cut out.
    Rectangle sides that are no Delaunay edges are halved until they are."""
    rng = np.random.default_rng(100 + seed)
    side = max(100.0, 71.0 * math.sqrt(count))
    lo, hi = (10, 60) if count > 8 else (10, 30)
    rects = [r.astype(np.float64) for r in random_rects(rng, side, side, count, lo, hi, 20000)]
    pts = [(0.0, 0.0), (side, 0.0), (side, side), (0.0, side)]
    want = []
    for r in rects:
        k = len(pts)
        pts += [tuple(p) for p in r]
        want += [(k, k + 1), (k + 1, k + 2), (k + 2, k + 3), (k + 3, k)]
    far = 1e4 * side
    jit = lambda n: rng.uniform(-1e-4, 1e-4, (n, 2))  # noqa: E731  (no four points on one circle)
    P = np.concatenate([[(-far, -far), (3 * far, -far), (-far, 3 * far)], np.array(pts) + jit(len(pts))])
    tri = np.array([[0, 1, 2]])

    def circles(t):
        a, b, c = P[t[:, 0]], P[t[:, 1]], P[t[:, 2]]
        d = 2 * ((b - a)[:, 0] * (c - a)[:, 1] - (b - a)[:, 1] * (c - a)[:, 0])
        b2, c2 = ((b - a) ** 2).sum(1), ((c - a) ** 2).sum(1)
        u = np.stack([(c - a)[:, 1] * b2 - (b - a)[:, 1] * c2, (b - a)[:, 0] * c2 - (c - a)[:, 0] * b2], 1) / d[:, None]
        return a + u, (u ** 2).sum(1)

    cen, rad = circles(tri)

    def insert(k):
        nonlocal tri, cen, rad
        bad = ((cen - P[k]) ** 2).sum(1) < rad
        e = tri[bad][:, [0, 1, 1, 2, 2, 0]].reshape(-1, 2)
        back = {(v, u) for u, v in e.tolist()}
        rim = np.array([(u, v) for u, v in e.tolist() if (u, v) not in back])
        new = np.column_stack([rim, np.full(len(rim), k)])
        c, r = circles(new)
        tri, cen, rad = np.concatenate([tri[~bad], new]), np.concatenate([cen[~bad], c]), np.concatenate([rad[~bad], r])

    for k in range(3, len(P)):
        insert(k)
    while True:
        have = {(min(u, v), max(u, v)) for u, v in (tri[:, [0, 1, 1, 2, 2, 0]].reshape(-1, 2) - 3).tolist()}
        gone = [w for w in want if (min(w), max(w)) not in have]
        if not gone:
            break
        for u, v in gone:
            k = len(pts)
            pts.append(tuple((np.array(pts[u]) + np.array(pts[v])) / 2))
            P = np.concatenate([P, np.array(pts[-1:]) + jit(1)])
            insert(k + 3)
            want.remove((u, v))
            want += [(u, k), (k, v)]
    tri = tri[(tri >= 3).all(1)] - 3
    vert = np.array(pts)
    mid = vert[tri].mean(1)
    keep = np.ones(len(tri), bool)
    for r in rects:
        keep &= ~((mid > r.min(0)) & (mid < r.max(0))).all(1)
    return _pack(vert.astype(np.float32), tri[keep])


_maps = {}


def _nodes(map, size, seed=0):
    """A map is loaded once by a program: kept per process."""
    key = (map, size, seed)
    if key not in _maps:
        if len(_maps) > 64:
            _maps.clear()
        _maps[key] = _maze(size) if map == "maze" else _rects(size, seed)
    return _maps[key]


def _points(nodes, n, rng):
    """n points uniform over the free area."""
    p1, p2, p3 = (nodes[f].astype(np.float64) for f in ("P1", "P2", "P3"))
    area = np.abs((p2 - p1)[:, 0] * (p3 - p1)[:, 1] - (p2 - p1)[:, 1] * (p3 - p1)[:, 0])
    k = np.searchsorted(np.cumsum(area), rng.random(n) * area.sum() * 0.999999)
    u = rng.random((n, 2))
    u = np.where(u.sum(1, keepdims=True) > 1, 1 - u, u) * 0.96 + 0.01
    return (p1[k] + u[:, :1] * (p2 - p1)[k] + u[:, 1:] * (p3 - p1)[k]).astype(np.float32)


# ---- preparation ------------------------------------------------------------

def _world(nodes, agents, c, rng):
    g = GMAPF()
    g.Init(make_config(max(1, agents), 2.0, 1.0, max(1, agents), c["T"], c["C"]))
    g.set_options(mode=c["mode"], path_smoothing=c["smooth"])
    g.FillMapManually(nodes)
    for p in _points(nodes, agents, rng):
        g.AddAgent(p)
    return g


def _some(rng, agents, share):
    k = int(round(agents * share))
    if k >= agents:
        return np.arange(agents, dtype=np.int32)
    return np.sort(rng.permutation(agents)[:k]).astype(np.int32)


def prepare(case, seed):
    c = case
    rng = np.random.default_rng([int(seed), c["agents"], c["size"]])
    if c["kind"] == "scenes":
        sizes = np.random.default_rng(c["scenes"])  # the scenes' agent counts are the case's, not the seed's
        share = np.diff(np.concatenate([[0], np.sort(sizes.integers(1, c["agents"], c["scenes"] - 1)), [c["agents"]]]))
        worlds, sets = [], []
        for k in range(c["scenes"]):
            nodes = _nodes("rects", max(4, c["size"] * (1 + k % 8) // 4), k % 8)
            # the agents a scene may hold, and its own retargets of every pass
            A = int(min(max(share[k], 1), 4 * len(nodes) + 64))
            worlds.append(_world(nodes, A, c, rng))
            sets.append((nodes, A))
        batch = SceneBatch(worlds)
        batch.ManualStart()
        for g, (nodes, A) in zip(worlds, sets):
            g.set_targets(np.arange(A, dtype=np.int32), _points(nodes, A, rng))
        for _ in range(2):
            batch.AsyncStep(DT)
            batch.WaitStepEnd()
        again = []
        for g, (nodes, A) in zip(worlds, sets):
            ids = _some(rng, A, c["retarget"])
            if len(ids):
                again.append((g, ids, _points(nodes, len(ids), rng)))
        return dict(case=c, batch=batch, again=again)

    nodes = _nodes(c["map"], c["size"])
    if c["kind"] in ("search", "noalloc"):
        n, N = c["agents"], len(nodes)
        stride = N if N < 40000 else N // 2
        g = GMAPF()
        g.Init(make_config(1, 2.0, 1.0, max(1, n), c["T"], c["C"]))
        g.FillMapManually(nodes)
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        s, t = (dev(g.locate(_points(nodes, n, rng)).astype(np.int32)) for _ in range(2))
        out = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2)]
        out.append(torch.full((n, stride), -1, dtype=torch.int32, device="cuda"))
        st = dict(case=c, n=n, N=N, stride=stride, s=s, t=t, out=out)
        if c["kind"] == "search":
            g.ManualStart()
            st["g"] = g
        else:
            st["nodes"] = dev(nodes.view(np.uint8))
        return st

    g = _world(nodes, c["agents"], c, rng)
    if c["kind"] == "serve":
        g.serve_start(0)
    else:
        g.ManualStart()
    if c["retarget"] < 1.0:  # everybody is on the way
        g.set_targets(np.arange(c["agents"], dtype=np.int32), _points(nodes, c["agents"], rng))
        for _ in range(2):
            g.AsyncStep(DT)
            g.WaitStepEnd()
    ids = _some(rng, c["agents"], c["retarget"])
    return dict(case=c, g=g, ids=ids, targets=_points(nodes, len(ids), rng))


# ---- one pass ---------------------------------------------------------------

def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "search":
        f, l, p = state["out"]
        st = state["g"].search_batch_device(state["s"].data_ptr(), state["t"].data_ptr(), state["n"], f.data_ptr(),
                                            l.data_ptr(), p.data_ptr(), state["stride"])
        return dict(found=f, lens=l, paths=p, stats=[st[k] for k in STATS[:7]])
    if kind == "noalloc":
        f, l, p = state["out"]
        lib = _lib.load()
        rc = lib.gmapf_search_batch_noalloc(state["nodes"].data_ptr(), state["N"], state["s"].data_ptr(),
                                            state["t"].data_ptr(), state["n"], c["T"], c["C"], 1.0, 0, f.data_ptr(),
                                            l.data_ptr(), p.data_ptr(), state["stride"],
                                            torch.cuda.current_stream().cuda_stream)
        if rc != 0:
            raise RuntimeError(lib.gmapf_last_error().decode())
        return dict(found=f, lens=l, paths=p)
    if kind == "scenes":
        b = state["batch"]
        for g, ids, pos in state["again"]:
            g.set_targets(ids, pos)
        b.AsyncStep(DT)
        b.WaitStepEnd()
        g = b.world
    elif kind == "serve":
        g = state["g"]
        g.serve_submit(state["ids"], state["targets"])
        g.serve_drain()
        g.AsyncStep(DT)
        g.WaitStepEnd()
    else:
        g = state["g"]
        if len(state["ids"]):
            g.set_targets(state["ids"], state["targets"])
        for _ in range(c["steps"]):
            g.AsyncStep(DT)
            g.WaitStepEnd()
    pos, st = g.agents()
    stats = g.last_stats()
    return dict(pos=pos, state=st, stats=[stats[k] for k in STATS])


def work(case):
    """Per expanded triangle: 12 B of neighbour ids and, per neighbour, 24 B (its centroid, visited word and
    record); per agent and frame: 80 B of position, step and path state; the map once.  Expanded per query: about a
    quarter of the triangles of a maze and a sixth of those between rectangles."""
    c = case
    if c["map"] == "maze":
        N, part = 4 * c["size"] ** 2, 0.25
    else:
        N, part = 8 * c["size"], 0.16
    queries = c["agents"] * (c["retarget"] if c["kind"] in ("frames", "scenes") else 1.0)
    moves = 0 if c["kind"] in ("search", "noalloc") else c["agents"] * c["steps"]
    return {"bytes": float(queries * (N * part * (12 + 2 * 24) + 32) + 80 * moves + 48 * N * c["scenes"]),
            "flops": float(queries * N * part * 2 * 6 + 40 * moves)}

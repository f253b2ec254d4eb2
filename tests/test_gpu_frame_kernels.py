"""The frame's own kernels at the sizes where they change form, against the oracle:
compaction at the edges of a block's step and of the cluster's, the grid's
buckets when cells hold more agents than fit, the funnel's window of 32 portals."""
import numpy as np
import pytest

import gmapf_b200 as G
from gmapf_b200.api import NODE_DTYPE
from gpu_util import close_rel

pytestmark = pytest.mark.gpu


def winding_map(rows, cols, side):
    """A corridor of rows x cols squares (two triangles each) that winds row by row."""
    quads, tris = [], []
    for y in range(rows):
        quads += [(x, y) for x in (range(cols) if y % 2 == 0 else range(cols - 1, -1, -1))]
    for x, y in quads:
        a, b, c, d = (x, y), (x + 1, y), (x + 1, y + 1), (x, y + 1)
        tris += [(a, b, c), (a, c, d)]
    out = np.zeros(2 * len(quads), NODE_DTYPE)
    nb = [[] for _ in range(len(out))]
    by_edge = {}
    for i, t in enumerate(tris):
        for f, v in zip(("P1", "P2", "P3"), t):
            out[f][i] = np.float32(v) * np.float32(side)
        for u, v in ((t[0], t[1]), (t[1], t[2]), (t[2], t[0])):
            by_edge.setdefault(frozenset((u, v)), []).append(i)
    for pair in by_edge.values():
        if len(pair) == 2 and abs(pair[0] // 2 - pair[1] // 2) <= 1:  # rows touch only where the corridor turns
            nb[pair[0]].append(pair[1])
            nb[pair[1]].append(pair[0])
    out["NeibsIdx"] = -1
    for i, l in enumerate(nb):
        out["NeibsIdx"][i, :len(l)] = l
    return out


def pair(oracle_mod, nodes, pos, T, Cap, P, radius=2.0, speed=1.0, smoothing=0):
    A = len(pos)
    g = G.GMAPF()
    g.Init(G.make_config(A, radius, speed, P, T, Cap))
    g.set_options(path_smoothing=smoothing)
    g.FillMapManually(nodes)
    om = oracle_mod.OMap(g.map_nodes())
    ow = oracle_mod.OWorld(om, A, radius, speed, P, T, Cap)
    ow.set_smoothing(smoothing)
    for p in pos:
        g.AddAgent(p)
        assert ow.add_agent(p[0], p[1]) >= 0
    return g, ow


def target(g, ow, ids, pos):
    g.set_targets(ids, pos)
    for i, p in zip(ids, pos):
        assert ow.set_target(int(i), p[0], p[1]) == 0


def step_and_compare(g, ow, dt):
    g.AsyncStep(dt)
    g.WaitStepEnd()
    ow.step(dt, 8)
    d, o = g.debug_agents(), ow.get()
    for k in ("state", "cur_node", "targ_node", "step_idx", "step_node", "path_len"):
        assert np.array_equal(d[k], o[k]), k
    assert close_rel(d["pos"], o["pos"])[0] and close_rel(d["step_pos"], o["step_pos"])[0]
    return d


def inside(nodes, n, rng):
    k = rng.integers(0, len(nodes), n)
    w = rng.dirichlet((1, 1, 1), n)[:, :, None] * 0.94 + 0.02
    return (w[:, 0] * nodes["P1"][k] + w[:, 1] * nodes["P2"][k] + w[:, 2] * nodes["P3"][k]).astype(np.float32)


@pytest.mark.parametrize("A", [3, 4093, 4096, 4097, 32768, 32771])
def test_compaction(oracle_mod, A):
    # a third of the agents retargeted, more than may search in one frame: the
    # requests are the first of them in id order, the rest the next frame's
    nodes = winding_map(2, 3, 40.0)
    rng = np.random.default_rng(A)
    P = max(1, A // 5)
    g, ow = pair(oracle_mod, nodes, inside(nodes, A, rng), 4, 8, P, radius=0.01)
    ids = np.nonzero(rng.random(A) < 0.34)[0].astype(np.int32)
    target(g, ow, ids, inside(nodes, len(ids), rng))
    for _ in range(3):
        step_and_compare(g, ow, 1.0)


@pytest.mark.parametrize("per_spot", [3, 5, 18, 40])
def test_crowded_cells(oracle_mod, per_spot):
    nodes = winding_map(3, 4, 60.0)
    rng = np.random.default_rng(per_spot)
    spots = inside(nodes, 6, rng)
    pos = (spots[:, None] + rng.normal(0, 0.8, (6, per_spot, 2))).reshape(-1, 2).astype(np.float32)
    probe = G.GMAPF()
    probe.Init(G.make_config(1, 2.0, 1.0, 1, 4, 8))
    probe.FillMapManually(nodes)
    pos = pos[probe.locate(pos) >= 0]
    pos = np.concatenate([pos, inside(nodes, 90, rng)])
    g, ow = pair(oracle_mod, nodes, pos, 8, 16, len(pos))
    target(g, ow, np.arange(len(pos), dtype=np.int32), inside(nodes, len(pos), rng))
    for _ in range(6):
        step_and_compare(g, ow, 0.5)


@pytest.mark.parametrize("smoothing", [1, 2])
@pytest.mark.parametrize("rows,cols", [(1, 9), (7, 5), (5, 33)])
def test_funnel_windows(oracle_mod, rows, cols, smoothing):
    # corridors of up to 330 triangles that turn back every `cols` squares:
    # corners inside a window, at its edges and far behind the walk
    nodes = winding_map(rows, cols, 10.0)
    rng = np.random.default_rng(rows)
    g, ow = pair(oracle_mod, nodes, inside(nodes, 24, rng), 8, 16, 24, radius=1.0, speed=4.0, smoothing=smoothing)
    target(g, ow, np.arange(24, dtype=np.int32), inside(nodes, 24, rng))
    for _ in range(40):
        step_and_compare(g, ow, 1.0)

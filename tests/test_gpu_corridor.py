"""The corridor kernel (long thin maps) against the oracle: bit-exact found flags,
lengths, paths and search counters, on maps whose searches take its slow paths:
random neighbour lists within a narrow window (asymmetric lists, repeated and
self neighbours, roots with one to three candidates, dropped queue entries)."""
import numpy as np
import pytest

import gmapf_b200 as G
from gmapf_b200.api import NODE_DTYPE

pytestmark = pytest.mark.gpu


def strip_map(n, window, seed):
    """n triangles; each lists up to three triangles at most `window` away."""
    rng = np.random.default_rng(seed)
    nodes = np.zeros(n, NODE_DTYPE)
    x = np.arange(n, dtype=np.float32)
    for f in ("P1", "P2", "P3"):
        nodes[f] = np.stack([x, np.zeros(n, np.float32)], 1) + rng.random((n, 2)).astype(np.float32)
    nb = np.full((n, 3), -1, np.int32)
    for i in range(n):
        d = int(rng.integers(1, 4))
        # (the next triangle is always listed: the map stays one long strip)
        nb[i, :d] = rng.integers(max(0, i - window), min(n, i + window + 1), d)
        nb[i, rng.integers(0, d)] = min(n - 1, i + 1)
    nodes["NeibsIdx"] = nb
    return nodes


def context(nodes, T, Cap, vm=0, mode=G.MODE_BATCHED):
    g = G.GMAPF()
    g.Init(G.make_config(4, 2.0, 1.0, 4, T, Cap))
    g.set_options(mode=mode, visited_mode=vm, promote_rounds=1 if vm == 4 else 0)
    g.FillMapManually(nodes)
    g.AddAgent(nodes["P1"][0])
    g.ManualStart()
    return g


def check(oracle_mod, g, nodes, s, t, T, Cap):
    om = oracle_mod.OMap(nodes)
    f, l, p, st = g.search_batch(s, t, len(nodes))
    of, ol, op, ost = om.search_batch(s, t, T, Cap)
    assert np.array_equal(f, of) and np.array_equal(l, ol)
    for i in np.nonzero(f)[0]:
        assert np.array_equal(p[i, :l[i]], op[i, :l[i]]), f"path {i} differs"
    for k in ("rounds", "expansions", "claims", "deg_sum"):
        assert st[k] == ost[k], k


@pytest.mark.parametrize("vm", [1, 4])
@pytest.mark.parametrize("T,Cap", [(2, 1), (2, 16), (4, 2), (8, 3), (8, 32), (16, 1), (16, 64), (32, 2), (32, 16)])
@pytest.mark.parametrize("n,window", [(1500, 3), (3000, 12)])
def test_strips(oracle_mod, n, window, T, Cap, vm):
    nodes = strip_map(n, window, seed=n + window)
    rng = np.random.default_rng(T * 100 + Cap)
    s, t = (rng.integers(0, n, 160).astype(np.int32) for _ in range(2))
    t[:40] = np.clip(s[:40] + rng.integers(-4, 5, 40), 0, n - 1)  # short searches: the sides meet at once
    g = context(nodes, T, Cap, vm)
    for _ in range(2):  # the second batch runs on the slots the first one used
        check(oracle_mod, g, nodes, s, t, T, Cap)


@pytest.mark.parametrize("mode", [G.MODE_BATCHED, G.MODE_PLAIN])
def test_queues_in_global_memory(oracle_mod, mode):
    # T=32, C=256: a warp's queues take 96 KB of shared memory, so the sizing
    # puts them in global memory
    nodes = strip_map(2000, 12, seed=5)
    rng = np.random.default_rng(6)
    s, t = (rng.integers(0, 2000, 300).astype(np.int32) for _ in range(2))
    check(oracle_mod, context(nodes, 32, 256, mode=mode), nodes, s, t, 32, 256)

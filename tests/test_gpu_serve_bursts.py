"""Bursts of retargets of any size: located on the device in portions, without a
wait for the searches in flight."""
import numpy as np
import pytest

import gmapf_b200 as G

pytestmark = pytest.mark.gpu


def test_growing_bursts_beside_long_searches():
    # searches of milliseconds; the second burst is larger than any before
    from test_gpu_frame_kernels import inside, winding_map
    nodes = winding_map(100, 100, 8.0)
    rng = np.random.default_rng(3)
    A = 6000
    g = G.GMAPF()
    g.Init(G.make_config(A, 0.1, 1.0, A, 8, 32))
    g.FillMapManually(nodes)
    for p in inside(nodes[:200], A, rng):
        g.AddAgent(p)
    g.serve_start(A)
    ids = np.arange(A, dtype=np.int32)
    g.serve_submit(ids[:8], inside(nodes[:200], 8, rng))
    g.serve_drain()
    goal = inside(nodes[-200:], A, rng)
    done, cuts = [], (0, 1100, 3200, A)
    for a, b in zip(cuts, cuts[1:]):  # each larger than the ones before
        g.serve_submit(ids[:1100], goal[:1100])
        before = g.serve_stats()["completed"]
        g.serve_submit(ids[a:b], goal[a:b])
        g.serve_poll()
        done.append(g.serve_stats()["completed"] - before)
        g.serve_drain()
    # (the host may be held up for as long as a search takes: once is enough)
    assert min(done[1:]) == 0, done
    assert g.serve_stats()["found"] == A + 8 + 3 * 1100


@pytest.mark.parametrize("n", [1023, 1024, 2100, 6500])
def test_bursts_of_any_size(oracle_mod, n):
    # more submissions than agents: an agent's last one counts
    from test_gpu_frame_kernels import inside, pair, winding_map
    nodes = winding_map(6, 9, 10.0)
    rng = np.random.default_rng(n)
    A = 1100
    start = inside(nodes, A, rng)
    g, _ = pair(oracle_mod, nodes, start, 8, 16, A, radius=0.1)
    g.serve_start(0)
    ids = rng.integers(0, A, n).astype(np.int32)
    goal = inside(nodes, n, rng)
    g.serve_submit(ids, goal)
    g.serve_drain()
    om = oracle_mod.OMap(g.map_nodes())
    last = {int(a): k for k, a in enumerate(ids)}
    agents = sorted(last)[::23]
    s = om.locate_batch(start[agents])
    t = om.locate_batch(goal[[last[a] for a in agents]])
    f, l, p, _ = om.search_batch(s, t, 8, 16)
    for k, a in enumerate(agents):
        gf, gl, gp = g.serve_result(a)
        assert gf == f[k] and gl == l[k] and np.array_equal(gp, p[k, :l[k]])

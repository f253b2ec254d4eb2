"""Frames of a serving context: they do not wait for the searches in flight, and
their compaction (made of smaller blocks while serving) is the frames' own."""
import numpy as np
import pytest

import gmapf_b200 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,Cap", [(8, 32), (32, 16)])
@pytest.mark.parametrize("A", [3000, 6000])
def test_frame_beside_long_searches(A, T, Cap):
    # every agent is sent from one end of a corridor of 20,000 triangles to the
    # other: some ten thousand rounds each (milliseconds), and a frame of a fraction
    # of one is over before the first search is
    from test_gpu_frame_kernels import inside, winding_map
    nodes = winding_map(100, 100, 8.0)
    rng = np.random.default_rng(A)
    g = G.GMAPF()
    g.Init(G.make_config(A, 0.1, 1.0, A, T, Cap))
    g.FillMapManually(nodes)
    for p in inside(nodes[:200], A, rng):
        g.AddAgent(p)
    g.serve_start(A)
    ids = np.arange(A, dtype=np.int32)
    g.serve_submit(ids[:8], inside(nodes[:200], 8, rng))
    g.serve_drain()
    g.AsyncStep(0.01)  # the first frame records its graph
    g.WaitStepEnd()
    done = []
    for k in range(3):  # (the host may be held up for as long as a search takes: once is enough)
        g.serve_submit(ids, inside(nodes[-200:] if k % 2 == 0 else nodes[:200], A, rng))
        g.AsyncStep(0.01)
        g.WaitStepEnd()
        g.serve_poll()
        done.append(g.serve_stats()["completed"] - 8 - k * A)
        g.serve_drain()
        if done[-1] == 0:
            break
    assert min(done) == 0, done
    assert g.serve_stats()["found"] == len(done) * A + 8


@pytest.mark.parametrize("A", [3, 1023, 1024, 1025, 8192, 8195, 16390])
def test_compaction_while_serving(oracle_mod, A):
    # a third of the agents retargeted, more than may search in one frame; a
    # frame before serving begins, two while it lasts and one after it
    from test_gpu_frame_kernels import inside, pair, step_and_compare, target, winding_map
    nodes = winding_map(2, 3, 40.0)
    rng = np.random.default_rng(A)
    P = max(1, A // 8)
    g, ow = pair(oracle_mod, nodes, inside(nodes, A, rng), 4, 8, P, radius=0.01)
    ids = np.nonzero(rng.random(A) < 0.34)[0].astype(np.int32)
    target(g, ow, ids, inside(nodes, len(ids), rng))
    step_and_compare(g, ow, 1.0)
    g.serve_start(0)
    step_and_compare(g, ow, 1.0)
    step_and_compare(g, ow, 1.0)
    g.serve_stop()
    step_and_compare(g, ow, 1.0)

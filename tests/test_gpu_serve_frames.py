"""Frames of a serving context: their compaction (made of smaller blocks while
serving) gives the requests of any other frame."""
import numpy as np
import pytest

import gmapf_b200 as G

pytestmark = pytest.mark.gpu


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

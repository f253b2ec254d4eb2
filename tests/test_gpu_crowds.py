"""Crowds in one place: grid cells that hold up to hundreds of agents, with few
and with many of them in reach, against the oracle's all-pairs collisions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("A,spread,radius", [(7, 0.1, 0.3), (60, 3.0, 0.3), (63, 1.0, 0.3), (601, 10.0, 0.3), (1500, 12.0, 0.2),
                                             (500, 6.0, 2.0), (300, 0.5, 1.0)])
def test_crowd_in_one_place(oracle_mod, A, spread, radius):
    from test_gpu_frame_kernels import inside, pair, step_and_compare, target, winding_map
    nodes = winding_map(3, 4, 60.0)
    rng = np.random.default_rng(A)
    th, r = rng.random(A) * 2 * np.pi, spread * np.sqrt(rng.random(A))
    pos = (np.stack([np.cos(th) * r, np.sin(th) * r], 1) + [95, 85]).astype(np.float32)
    pos[rng.integers(0, A, A // 10)] = inside(nodes, A // 10, rng)  # some elsewhere
    g, ow = pair(oracle_mod, nodes, pos, 8, 16, A, radius=radius)
    target(g, ow, np.arange(A, dtype=np.int32), (pos * 0.1 + [85, 76]).astype(np.float32))
    for _ in range(6):
        step_and_compare(g, ow, 0.4)

"""Searches without allocation whose two ends have neighbour lists of different
shape: one with three neighbours, one with ids outside the navmesh among its
three, so that the first round's candidates are not lined up by place."""
import ctypes as C

import numpy as np
import pytest

from gmapf_b200.api import NODE_DTYPE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,Cap", [(2, 3), (4, 16), (8, 32), (16, 2), (32, 16)])
@pytest.mark.parametrize("hole", [0, 1, 2])
def test_ends_with_a_hole_in_their_list(lib, oracle_mod, T, Cap, hole):
    import torch
    # a sheet of triangles, six around every corner: most have three neighbours
    side, q = 20, 400
    n = 2 * side * side
    rng = np.random.default_rng(hole)
    nodes = np.zeros(n, NODE_DTYPE)
    y, x, up = (v.ravel() for v in np.mgrid[0:side, 0:side, 0:2])
    for f, dx, dy in (("P1", 0, 0), ("P2", 1, up), ("P3", 1 - up, 1)):
        nodes[f] = np.stack([x + dx, y + dy], 1) * 3 + rng.random((n, 2)) * 0.2
    near = np.stack([np.arange(n) ^ 1, np.where(up, ((y + 1) * side + x) * 2, (y * side + x - 1) * 2 + 1),
                     np.where(up, (y * side + x + 1) * 2, ((y - 1) * side + x) * 2 + 1)], 1)
    there = np.stack([np.ones(n, bool), np.where(up, y + 1 < side, x > 0), np.where(up, x + 1 < side, y > 0)], 1)
    order = np.argsort(rng.random((n, 3)) + ~there, axis=1)  # in any order, those that exist first
    nb = np.take_along_axis(np.where(there, near, -1), order, 1)
    holed = (np.arange(n) % 2 == 1) & (nb[:, hole] >= 0)
    same = nodes.copy()
    nodes["NeibsIdx"] = np.where(holed[:, None] & (np.arange(3) == hole), n + 5, nb)
    same["NeibsIdx"] = np.where(holed[:, None] & (np.arange(3) == hole), np.arange(n)[:, None], nb)
    a, b = rng.integers(0, n // 2, q) * 2, rng.integers(0, n // 2, q) * 2 + 1
    flip = np.arange(q) % 4 == 0
    s, t = (np.where(flip, b, a).astype(np.int32), np.where(flip, a, b).astype(np.int32))
    # (a triangle that lists itself claims nothing there: as an id outside the navmesh)
    of, ol, op, _ = oracle_mod.OMap(same).search_batch(s, t, T, Cap)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    d_nodes, d_s, d_t = dev(nodes.view(np.uint8)), dev(s), dev(t)
    f, l = (torch.full((q,), -7, dtype=torch.int32, device="cuda") for _ in range(2))
    p = torch.full((q, n), -7, dtype=torch.int32, device="cuda")
    rc = lib.gmapf_search_batch_noalloc(d_nodes.data_ptr(), n, d_s.data_ptr(), d_t.data_ptr(), q, T, Cap,
                                        C.c_float(1.0), 0, f.data_ptr(), l.data_ptr(), p.data_ptr(), n,
                                        C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert rc == 0
    gf, gl, gp = f.cpu().numpy(), l.cpu().numpy(), p.cpu().numpy()
    assert np.array_equal(gf, of) and np.array_equal(gl, ol) and of.sum() > q // 4
    for i in np.nonzero(gf)[0]:
        assert np.array_equal(gp[i, :gl[i]], op[i, :gl[i]]), f"path {i}"

"""Few queries on a large navmesh, without allocation: short ones are answered in
the record form, longer ones by the log form after it.  Against the oracle, and
against the same queries in a call that takes the log form for all of them."""
import ctypes as C

import numpy as np
import pytest

from gmapf_b200.api import NODE_DTYPE

pytestmark = pytest.mark.gpu


def sheet(side):
    """side x side squares, two triangles each."""
    n = 2 * side * side
    nodes = np.zeros(n, NODE_DTYPE)
    y, x, up = (v.ravel() for v in np.mgrid[0:side, 0:side, 0:2])
    for f, dx, dy in (("P1", 0, 0), ("P2", 1, up), ("P3", 1 - up, 1)):
        nodes[f] = np.stack([x + dx, y + dy], 1) * 3.0
    near = np.stack([np.arange(n) ^ 1, np.where(up, ((y + 1) * side + x) * 2, (y * side + x - 1) * 2 + 1),
                     np.where(up, (y * side + x + 1) * 2, ((y - 1) * side + x) * 2 + 1)], 1)
    there = np.stack([np.ones(n, bool), np.where(up, y + 1 < side, x > 0), np.where(up, x + 1 < side, y > 0)], 1)
    order = np.argsort(~there, axis=1, kind="stable")
    nodes["NeibsIdx"] = np.take_along_axis(np.where(there, near, -1), order, 1)
    return nodes


def run(lib, nodes, d_nodes, s, t, T, Cap, limit=0, stride=4000):
    import torch
    q = len(s)
    d_s, d_t = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (s, t))
    f, l = (torch.full((q,), -7, dtype=torch.int32, device="cuda") for _ in range(2))
    p = torch.full((q, stride), -7, dtype=torch.int32, device="cuda")
    rc = lib.gmapf_search_batch_noalloc(d_nodes.data_ptr(), len(nodes), d_s.data_ptr(), d_t.data_ptr(), q, T, Cap,
                                        C.c_float(1.0), limit, f.data_ptr(), l.data_ptr(), p.data_ptr(), stride,
                                        C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert rc == 0
    return f.cpu().numpy(), l.cpu().numpy(), p.cpu().numpy()


@pytest.mark.parametrize("T,Cap", [(2, 3), (8, 32), (16, 4), (32, 16)])
@pytest.mark.parametrize("side", [180, 256, 300])  # 64,800, 131,072 and 180,000 triangles
def test_few_queries_on_a_large_navmesh(lib, oracle_mod, side, T, Cap):
    import torch
    nodes = sheet(side)
    n = len(nodes)
    d_nodes = torch.from_numpy(nodes.view(np.uint8)).cuda()
    rng = np.random.default_rng(side + T)
    om = oracle_mod.OMap(nodes)
    for q in (1, 2, 11, 12, 15, 16, 22, 23, 30, 31):
        s = rng.integers(0, n, q)
        hop = rng.choice([0, 2, 6, 14, 30, 31, 32, 33, 34, 60, 400], q)  # squares away
        t = np.clip(s + 2 * hop * rng.choice([-1, 1, side], q), 0, n - 1)
        s, t = s.astype(np.int32), t.astype(np.int32)
        ok = np.ones(q, bool)
        if q > 10:
            s[3], t[7], ok[3], ok[7] = -1, n, False, False
        of, ol, op, _ = om.search_batch(np.where(ok, s, 0), np.where(ok, t, 0), T, Cap, path_stride=4000)
        for _ in range(2):
            f, l, p = run(lib, nodes, d_nodes, s, t, T, Cap)
            assert np.array_equal(f[ok], of[ok]) and np.array_equal(l[ok], ol[ok])
            assert np.all(f[~ok] == -1) and np.all(l[~ok] == 0)
            for i in np.nonzero(ok & (f == 1))[0]:
                assert np.array_equal(p[i, :l[i]], op[i, :l[i]])
        if q == 11:  # round limits below, at and above the record form's share
            more = [np.resize(x, 200) for x in (s, t)]
            for limit in (3, 7, 8, 9, 15, 16, 17, 40):
                f, l, _ = run(lib, nodes, d_nodes, s, t, T, Cap, limit)
                F, L, _ = run(lib, nodes, d_nodes, *more, T, Cap, limit)
                assert np.array_equal(f, F[:q]) and np.array_equal(l, L[:q])

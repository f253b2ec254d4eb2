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


@pytest.mark.parametrize("T,Cap", [(2, 3), (8, 32), (16, 1), (32, 16)])
def test_noalloc_log_form(lib, oracle_mod, T, Cap):
    # caller-provided records: asymmetric lists, and neighbour ids outside the
    # navmesh, which are no candidates (as if the triangle listed itself)
    import ctypes as C
    import torch
    n = 1200
    nodes = strip_map(n, 12, seed=9)
    rng = np.random.default_rng(10)
    same = nodes.copy()
    for i in rng.integers(0, n, 150):
        k = int(rng.integers(0, 3))
        if nodes["NeibsIdx"][i, k] >= 0 and nodes["NeibsIdx"][i, k] != min(n - 1, i + 1):
            nodes["NeibsIdx"][i, k] = [-9, n, 2**31 - 1][i % 3]
            same["NeibsIdx"][i, k] = i
    s, t = (rng.integers(0, n, 200).astype(np.int32) for _ in range(2))
    s[7], t[9], t[11] = -1, n, s[11]
    ok = np.ones(200, bool)
    ok[[7, 9]] = False
    of, ol, op, _ = oracle_mod.OMap(same).search_batch(np.where(ok, s, 0), np.where(ok, t, 1), T, Cap)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    d_nodes, d_s, d_t = dev(nodes.view(np.uint8)), dev(s), dev(t)
    f, l = (torch.full((200,), -7, dtype=torch.int32, device="cuda") for _ in range(2))
    p = torch.full((200, n), -7, dtype=torch.int32, device="cuda")
    for _ in range(2):
        rc = lib.gmapf_search_batch_noalloc(d_nodes.data_ptr(), n, d_s.data_ptr(), d_t.data_ptr(), 200, T, Cap,
                                            C.c_float(1.0), 0, f.data_ptr(), l.data_ptr(), p.data_ptr(), n,
                                            C.c_void_p(torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert rc == 0
        gf, gl, gp = f.cpu().numpy(), l.cpu().numpy(), p.cpu().numpy()
        assert np.array_equal(gf[~ok], [-1, -1]) and np.array_equal(gl[~ok], [0, 0])
        assert np.array_equal(gf[ok], of[ok]) and np.array_equal(gl[ok], ol[ok])
        for i in np.nonzero(ok & (gf == 1))[0]:
            assert np.array_equal(gp[i, :gl[i]], op[i, :gl[i]])


@pytest.mark.parametrize("n", [0x7fc0, 0x7fc1])
def test_noalloc_log_entry_sizes(lib, oracle_mod, n):
    # the largest navmesh with 6-byte log entries and the smallest with 8: ids,
    # log places and depths (searches of a triangle nobody lists run to the
    # strip's other end) up to the ends of their fields
    import ctypes as C
    import torch
    T, Cap, q = 8, 32, 40
    nodes = strip_map(n, 2, seed=13)
    nb = nodes["NeibsIdx"]
    nb[nb == n - 2] = n - 1
    nb[n - 2] = -1
    rng = np.random.default_rng(14)
    s, t = (rng.integers(0, n, q).astype(np.int32) for _ in range(2))
    s[:4], t[:4] = [0, 1, n - 1, n - 1], [n - 2, n - 1, 0, n - 2]
    of, ol, op, _ = oracle_mod.OMap(nodes).search_batch(s, t, T, Cap)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    d_nodes, d_s, d_t = dev(nodes.view(np.uint8)), dev(s), dev(t)
    f, l = (torch.full((q,), -7, dtype=torch.int32, device="cuda") for _ in range(2))
    p = torch.full((q, n), -7, dtype=torch.int32, device="cuda")
    rc = lib.gmapf_search_batch_noalloc(d_nodes.data_ptr(), n, d_s.data_ptr(), d_t.data_ptr(), q, T, Cap,
                                        C.c_float(1.0), 0, f.data_ptr(), l.data_ptr(), p.data_ptr(), n,
                                        C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert rc == 0
    gf, gl, gp = f.cpu().numpy(), l.cpu().numpy(), p.cpu().numpy()
    assert np.array_equal(gf, of) and np.array_equal(gl, ol) and gl.max() > n // 4
    for i in np.nonzero(gf)[0]:
        assert np.array_equal(gp[i, :gl[i]], op[i, :gl[i]])


def test_scene_batch_and_serving_on_corridors(oracle_mod):
    # two winding corridors stepped as one batch, then one of them served: the
    # corridor kernel with global ids, and on the serving streams
    from test_gpu_frame_kernels import inside, pair, step_and_compare, target, winding_map
    maps = [winding_map(9, 40, 8.0), winding_map(20, 18, 9.0)]
    rng = np.random.default_rng(12)
    sets = []
    for nodes in maps:
        g, ow = pair(oracle_mod, nodes, inside(nodes, 50, rng), 8, 16, 50, radius=1.0)
        sets.append((g, ow, nodes))
    batch = G.SceneBatch([g for g, _, _ in sets])
    batch.ManualStart()
    assert batch.world.search_shape()["T"] == 8
    for frame in range(4):
        if frame % 2 == 0:
            for g, ow, nodes in sets:
                target(g, ow, np.arange(50, dtype=np.int32), inside(nodes, 50, rng))
        batch.AsyncStep(0.5)
        batch.WaitStepEnd()
        for g, ow, _ in sets:
            ow.step(0.5, 4)
            d, o = g.debug_agents(), ow.get()
            for k in ("state", "path_len", "step_idx"):
                assert np.array_equal(d[k], o[k]), k
    nodes = maps[1]
    start, goal = inside(nodes, 1500, rng), inside(nodes, 1500, rng)
    g, _ = pair(oracle_mod, nodes, start, 8, 16, 1500, radius=0.1)
    g.serve_start(0)
    g.serve_submit(np.arange(1500, dtype=np.int32), goal)
    g.serve_drain()
    om = oracle_mod.OMap(g.map_nodes())
    s, t = om.locate_batch(start), om.locate_batch(goal)
    f, l, p, _ = om.search_batch(s, t, 8, 16)
    for a in range(0, 1500, 37):
        gf, gl, gp = g.serve_result(a)
        assert gf == f[a] and gl == l[a] and np.array_equal(gp, p[a, :l[a]])

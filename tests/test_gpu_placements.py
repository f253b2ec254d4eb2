"""Which visited placements a corridor map takes: the same that any other map of
its size takes, whichever kernel searches it."""
import numpy as np
import pytest

import gmapf_b200 as G
from gmapf_b200.api import NODE_DTYPE

pytestmark = pytest.mark.gpu


def long_strip(n):
    """n triangles in a row, each next to the one before and the one after."""
    nodes = np.zeros(n, NODE_DTYPE)
    x = np.arange(n, dtype=np.float32)
    for f, dx, dy in (("P1", 0, 0), ("P2", 1, 0), ("P3", 0.5, 1)):
        nodes[f] = np.stack([x * 0.5 + dx, (x % 2) + dy * (1 - 2 * (x % 2))], 1)
    i = np.arange(n)
    nodes["NeibsIdx"] = np.stack([np.where(i > 0, i - 1, 1), np.where((i > 0) & (i < n - 1), i + 1, -1),
                                  np.full(n, -1)], 1)
    return nodes


def start(nodes, T, Cap, **options):
    g = G.GMAPF()
    g.Init(G.make_config(1, 2.0, 1.0, 1, T, Cap))
    g.set_options(**options)
    g.FillMapManually(nodes)
    g.ManualStart()
    return g


@pytest.mark.parametrize("vm", [1, 4])
def test_bitmap_that_just_fits(oracle_mod, vm):
    # 231,252 bytes of bitmap: room beside search.cu's share of T=2, C=1 (112
    # bytes), not beside corridor.cu's (1.6 KB)
    n = 925_000
    nodes = long_strip(n)
    rng = np.random.default_rng(vm)
    s = rng.integers(3000, n - 3000, 6).astype(np.int32)
    t = (s + rng.integers(-2000, 2000, 6)).astype(np.int32)
    g = start(nodes, 2, 1, visited_mode=vm)
    assert g.search_shape()["visited_mode"] == vm
    f, l, p, _ = g.search_batch(s, t, 4000)
    of, ol, op, _ = oracle_mod.OMap(nodes).search_batch(s, t, 2, 1)
    assert np.array_equal(f, of) and np.array_equal(l, ol) and f.all()
    for i in range(len(s)):
        assert np.array_equal(p[i, :l[i]], op[i, :l[i]])


@pytest.mark.parametrize("vm", [1, 4])
def test_queues_that_leave_no_room(vm):
    # 196,608 bytes of queues and 50,000 of bitmap
    with pytest.raises(G.GMAPFError, match="E_CAPACITY"):
        start(long_strip(200_000), 32, 512, visited_mode=vm)
    assert start(long_strip(200_000), 32, 512).search_shape()["slots"] > 0


@pytest.mark.parametrize("options", [{}, dict(autotune=True), dict(visited_mode=4)])
def test_search_memory_within_its_budget(options):
    # T=32, C=256: 98,304 bytes of queues to 32,000 of claim log in a slot
    import torch
    nodes, budget = long_strip(2000), 64 << 20
    start(nodes, 32, 256, **options).close()  # (what the process keeps is there)

    def held(budget):
        before = torch.cuda.mem_get_info()[0]
        g = start(nodes, 32, 256, search_mem_budget=budget, **options)
        used = before - torch.cuda.mem_get_info()[0]
        g.close()
        return used

    assert held(budget) - held(1 << 20) <= budget + (8 << 20)  # (2 MiB granules)


@pytest.mark.parametrize("P,one_chunk", [(3000, True), (4000, True), (16384, False)])
def test_plain_form_takes_the_kernel_with_fewer_chunks(oracle_mod, P, one_chunk):
    # T=8: search.cu's kernel has 28 warps per SM (4,144 slots), corridor.cu's 24 (3,552)
    nodes = long_strip(2700)
    g = G.GMAPF()
    g.Init(G.make_config(1, 2.0, 1.0, P, 8, 32))
    g.set_options(mode=G.MODE_PLAIN)
    g.FillMapManually(nodes)
    g.ManualStart()
    assert (g.search_shape()["slots"] >= P) == one_chunk
    rng = np.random.default_rng(P)
    s, t = (rng.integers(0, len(nodes), 300).astype(np.int32) for _ in range(2))
    f, l, p, _ = g.search_batch(s, t, len(nodes))
    of, ol, op, _ = oracle_mod.OMap(nodes).search_batch(s, t, 8, 32)
    assert np.array_equal(f, of) and np.array_equal(l, ol)
    for i in np.nonzero(f)[0]:
        assert np.array_equal(p[i, :l[i]], op[i, :l[i]])

"""Visited placement 4 in the corridor kernel where a block has no room of its own
for a bitmap: a long search moves its bitmap into the shares of its block's finished
warps, and its queues and frontier with it when its own share is among them.
Against the oracle, with queues in shared and in global memory, in batches with a
warp for every request and in batches that the queue feeds."""
import ctypes as C

import numpy as np
import pytest

import gmapf_b200 as G

pytestmark = pytest.mark.gpu


def no_room_of_its_own(lib, n, T, Cap, threads):
    """Both forms of the queues: a block with room for a whole bitmap more would
    cost the SM a block, so the sizing leaves it out."""
    blocks = lib._ZN10gmapf_b20026corridor_max_blocks_per_smEiiiiibb
    blocks.argtypes = [C.c_int] * 5 + [C.c_bool] * 2
    words = ((n + 15) // 16 + 3) & ~3
    return all(0 < blocks(T, Cap, threads, 4, words, q, False) > blocks(T, Cap, threads, 4, words, q, True)
               for q in (False, True))


def compare(oracle_mod, g, nodes, T, Cap):
    n, shape = len(nodes), g.search_shape()
    om = oracle_mod.OMap(nodes)
    rng = np.random.default_rng(n)
    for q in (shape["slots"] // 2, shape["slots"] + 700):
        # in every block a few searches of thousands of rounds among short ones
        hops = np.where(rng.random(q) < 0.2, rng.integers(2500, 3900, q), rng.integers(1, 40, q))
        s = rng.integers(4000, n - 4000, q)
        t = s + hops * rng.choice([-1, 1], q)
        s, t = s.astype(np.int32), t.astype(np.int32)
        f, l, p, st = g.search_batch(s, t, 4000)
        of, ol, op, ost = om.search_batch(s, t, T, Cap, path_stride=4000)
        assert st["promoted"] > 0
        assert np.array_equal(f, of) and np.array_equal(l, ol) and f.mean() > 0.9
        for i in np.nonzero(f)[0]:
            assert np.array_equal(p[i, :l[i]], op[i, :l[i]]), f"path {i} differs"
        for k in ("rounds", "expansions", "claims", "deg_sum"):
            assert st[k] == ost[k], k


def started(nodes, T, Cap, **options):
    g = G.GMAPF()
    g.Init(G.make_config(1, 2.0, 1.0, 1, T, Cap))
    g.set_options(visited_mode=4, promote_rounds=1, **options)
    g.FillMapManually(nodes)
    g.ManualStart()
    assert g.search_shape()["visited_mode"] == 4
    return g


@pytest.mark.parametrize("T,Cap,threads,n", [(8, 32, 64, 90_000), (8, 32, 128, 126_000), (32, 16, 64, 90_000),
                                             (32, 16, 128, 140_000), (32, 16, 256, 180_000), (2, 4, 256, 270_000)])
def test_move_into_finished_warps_shares(lib, oracle_mod, T, Cap, threads, n):
    from test_gpu_placements import long_strip
    nodes = long_strip(n)
    g = started(nodes, T, Cap, block_threads=threads)
    assert g.search_shape()["block_threads"] == threads
    assert no_room_of_its_own(lib, n, T, Cap, threads)
    compare(oracle_mod, g, nodes, T, Cap)


@pytest.mark.parametrize("T,Cap", [(8, 32), (32, 16)])
def test_room_of_its_own(lib, oracle_mod, T, Cap):
    # the same batches where every block has room for a bitmap of its own: taken
    # while the block's others run, and by the tail of a batch that the queue feeds
    from test_gpu_placements import long_strip
    n = 30_000
    g = started(long_strip(n), T, Cap, block_threads=256)
    assert not no_room_of_its_own(lib, n, T, Cap, 256)
    compare(oracle_mod, g, long_strip(n), T, Cap)

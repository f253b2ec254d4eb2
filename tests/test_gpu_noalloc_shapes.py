"""Searches without allocation with one queue capacity after the other, in the
record form (few short queries on a large navmesh)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [2, 8, 32])
def test_capacities_in_any_order(lib, oracle_mod, T):
    import torch
    from test_gpu_noalloc_few import run, sheet
    nodes = sheet(260)
    d_nodes = torch.from_numpy(nodes.view(np.uint8)).cuda()
    om = oracle_mod.OMap(nodes)
    s = np.array([1000, 70_000], np.int32)
    t = s + np.array([4, 1042], np.int32)
    for Cap in (64, 5, 64, 128, 16, 64, 128):
        f, l, p = run(lib, nodes, d_nodes, s, t, T, Cap)
        of, ol, op, _ = om.search_batch(s, t, T, Cap, path_stride=4000)
        assert np.array_equal(f, of) and np.array_equal(l, ol)
        for i in np.nonzero(f)[0]:
            assert np.array_equal(p[i, :l[i]], op[i, :l[i]])

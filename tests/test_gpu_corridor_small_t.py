"""The corridor kernel with two and four threads per agent, which it serves only in
long corridors (1,000 levels), against the oracle, and that it is the one that ran."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vm", [1, 4])
@pytest.mark.parametrize("T,Cap", [(2, 1), (2, 16), (4, 2), (4, 64), (8, 3), (16, 1), (32, 2)])
def test_long_strips(oracle_mod, T, Cap, vm):
    import torch
    from test_gpu_corridor import check, context, strip_map
    n = 7000
    nodes = strip_map(n, 12, seed=31)
    rng = np.random.default_rng(T * 100 + Cap)
    s, t = (rng.integers(0, n, 160).astype(np.int32) for _ in range(2))
    t[:40] = np.clip(s[:40] + rng.integers(-4, 5, 40), 0, n - 1)
    g = context(nodes, T, Cap, vm)
    # 80 registers: 24 warps per SM (search.cu's kernel has 28 at T <= 8)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if T <= 8:
        assert g.search_shape()["slots"] == 24 * sms
    for _ in range(2):
        check(oracle_mod, g, nodes, s, t, T, Cap)

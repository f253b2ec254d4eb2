"""A start that fails leaves nothing behind for the next one of the same context."""
import os
import subprocess
from pathlib import Path

import numpy as np
import pytest

import gmapf_b200 as G

ROOT = Path(__file__).resolve().parents[1]


def test_device_free_forgets_what_a_start_set(lib, tmp_path):
    exe = tmp_path / "device_free_check"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    pkg = ROOT / "gmapf_b200"
    subprocess.run(["g++", "-std=c++17", "-I", str(pkg / "csrc"), "-I", str(ROOT / "include"), "-I", cuda + "/include",
                    str(ROOT / "tests" / "cpp" / "device_free_check.cpp"), str(pkg / "libgmapf_b200.so"),
                    f"-Wl,-rpath,{pkg}", "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("second", [dict(mode=G.MODE_PLAIN), dict(order_by_estimate=False)])
def test_frames_after_a_failed_start(oracle_mod, second):
    # the failed start asks for the request order's buffers, the second does not
    from test_gpu_frame_kernels import inside, step_and_compare, target, winding_map
    nodes = winding_map(6, 9, 10.0)
    rng = np.random.default_rng(21)
    g = G.GMAPF()
    g.Init(G.make_config(30, 1.0, 1.0, 30, 8, 16))
    g.set_options(search_mem_budget=1)
    g.FillMapManually(nodes)
    om = oracle_mod.OMap(g.map_nodes())
    ow = oracle_mod.OWorld(om, 30, 1.0, 1.0, 30, 8, 16)
    pos = inside(nodes, 30, rng)
    for k, p in enumerate(pos):
        if k in (0, 10):
            with pytest.raises(G.GMAPFError, match="E_CAPACITY"):
                g.ManualStart()
        g.AddAgent(p)
        assert ow.add_agent(p[0], p[1]) >= 0
    g.set_options(search_mem_budget=0, **second)
    g.ManualStart()
    target(g, ow, np.arange(30, dtype=np.int32), inside(nodes, 30, rng))
    for _ in range(4):
        step_and_compare(g, ow, 0.5)
    s, t = (rng.integers(0, len(nodes), 50).astype(np.int32) for _ in range(2))
    f, l, p, _ = g.search_batch(s, t, len(nodes))
    of, ol, op, _ = om.search_batch(s, t, 8, 16)
    assert np.array_equal(f, of) and np.array_equal(l, ol)
    for i in np.nonzero(f)[0]:
        assert np.array_equal(p[i, :l[i]], op[i, :l[i]])

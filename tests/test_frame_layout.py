"""Where a frame's counters and statistics lie (a host program on the library's
own header)."""
import os
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_counters_and_statistics_share_no_line(tmp_path):
    exe = tmp_path / "frame_layout_check"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT / "gmapf_b200" / "csrc"), "-I", str(ROOT / "include"),
                    "-I", cuda + "/include", str(ROOT / "tests" / "cpp" / "frame_layout_check.cpp"), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout

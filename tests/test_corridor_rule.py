"""Which kernel searches a map (the library's own rule, called by a host program)."""
import os
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_corridor_rule(lib, tmp_path):
    exe = tmp_path / "corridor_rule_check"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    pkg = ROOT / "gmapf_b200"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(pkg / "csrc"), "-I", str(ROOT / "include"), "-I",
                    cuda + "/include", str(ROOT / "tests" / "cpp" / "corridor_rule_check.cpp"),
                    str(pkg / "libgmapf_b200.so"), f"-Wl,-rpath,{pkg}", "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr

"""The captured wave graphs (vork_b200/csrc/vkb_graphs.h): keys and bounds, no GPU."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_wave_graph_keys_and_bounds(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("needs g++")
    exe = tmp_path / "graphs_harness"
    subprocess.run([gxx, "-O1", "-std=c++17", "-Wall", f"-I{ROOT / 'vork_b200' / 'csrc'}", str(ROOT / "tests" / "graphs_harness.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "OK", r.stdout + r.stderr

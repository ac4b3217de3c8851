"""The device buffers kept between objects (vork_b200/csrc/vkb_pool.h), no GPU."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_kept_buffers(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("needs g++")
    exe = tmp_path / "pool_harness"
    subprocess.run([gxx, "-O1", "-std=c++17", "-Wall", "-pthread", f"-I{ROOT / 'vork_b200' / 'csrc'}", str(ROOT / "tests" / "pool_harness.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "OK", r.stdout + r.stderr


def test_device_memory_comes_from_one_place():
    # An allocation that goes past device_alloc fails while pools hold memory idle.
    calls = [m.group(0) for p in sorted((ROOT / "vork_b200" / "csrc").glob("*")) for m in re.finditer(r"cudaMalloc\w*\(", re.sub(r"//[^\n]*|\"[^\"\n]*\"", "", p.read_text()))]
    assert calls == ["cudaMalloc("]

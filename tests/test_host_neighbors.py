"""CPU test of the neighbour search (common.cuh) on axes of 1 to 5 points: too
few points give a status, whatever the label, and nothing past an axis is read."""
import os
import subprocess

from test_host_memory import HERE, _cuda_include


def test_short_axes(tmp_path):
    out = str(tmp_path / "neighbors_cases")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", "-I" + _cuda_include(),
                    os.path.join(HERE, "neighbors_cases.cpp"), "-o", out], check=True)
    r = subprocess.run([out], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr[:2000]

"""CPU test of the allocation-free chi2's scratch layout (noalloc_layout.h):
every label count that is accepted fits the static array."""
import os
import subprocess

from test_host_memory import HERE, _cuda_include


def test_accepted_label_counts_fit_the_scratch(tmp_path):
    out = str(tmp_path / "noalloc_cases")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + _cuda_include(), os.path.join(HERE, "noalloc_cases.cpp"), "-o", out],
                   check=True)
    r = subprocess.run([out], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout

"""CPU tests of the engine's memory (hostmem.h): what happens when an allocation,
a page-locked buffer or a thread cannot be had.  hostmem_cases.cpp compiles the
header against a stand-in for the CUDA runtime whose calls fail on demand."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def _cuda_include():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")


@pytest.fixture(scope="session")
def binary(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("hostmem") / "hostmem_cases")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-pthread", "-I" + _cuda_include(),
                    os.path.join(HERE, "hostmem_cases.cpp"), "-o", out], check=True)
    return out


def _run(binary, case):
    r = subprocess.run([binary, case], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr or r.returncode


@pytest.mark.parametrize("case", ["flush_while_contexts_are_looked_up", "context_without_memory"])
def test_pool_is_given_back_when_memory_runs_out(binary, case):
    _run(binary, case)


def test_context_that_failed_is_made_again(binary):
    _run(binary, "context_made_again")


def test_copies_go_on_without_page_locked_memory(binary):
    _run(binary, "copies_without_staging")


def test_copy_threads_without_host_memory(binary):
    _run(binary, "threads_without_host_memory")


def test_scratch_that_fits_exactly(binary):
    _run(binary, "exact_fits")


def test_graph_captures_are_alone(binary):
    _run(binary, "captures_are_alone")


def test_uploads_are_waited_for(binary):
    _run(binary, "uploads_are_waited_for")

"""Host-side pieces of the library's internals, compiled alone and run without a GPU."""
import os
import subprocess

import pytest

from cxx_util import CXX_DIR, ROOT, compiler

pytestmark = pytest.mark.skipif(compiler() is None, reason="no C++ compiler")

CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def run_program(name, tmp_path, units=()):
    """Compiles tests/cxx/<name>.cpp and these of the library's host units
    against the internal headers (no CUDA runtime linked) and returns its
    output."""
    out = str(tmp_path / name)
    cmd = [compiler(), "-std=c++17", "-O1", "-Wall", "-I",
           os.path.join(ROOT, "unap_gb300", "csrc"), "-I", CUDA_INCLUDE,
           os.path.join(CXX_DIR, f"{name}.cpp"),
           *(os.path.join(ROOT, "unap_gb300", "csrc", u) for u in units), "-o", out, "-pthread"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([out], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


def test_row_counts_of_long_rows(tmp_path):
    assert "ok" in run_program("row_info", tmp_path)


def test_failed_allocation_gives_the_workspace_pool_back(tmp_path):
    assert "ok" in run_program("alloc_retry", tmp_path)


def test_failed_allocation_leaves_nothing_behind(tmp_path):
    assert "ok" in run_program("alloc_state", tmp_path, units=["flow_ring.cpp"])


def test_growing_ring_keeps_its_error_word(tmp_path):
    assert "ok" in run_program("ring_error_word", tmp_path, units=["flow_ring.cpp"])


def test_sweeps_keep_what_their_launches_write(tmp_path):
    assert "ok" in run_program("ring_storage", tmp_path, units=["flow_ring.cpp"])


def test_where_setup_runs_by_kernels(tmp_path):
    assert "ok" in run_program("setup_limits", tmp_path)

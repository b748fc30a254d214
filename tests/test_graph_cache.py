"""The cache of captured solves (gpumatting_b200/csrc/gm_graph_cache.h): its
error paths, with a fake capture (tests/c/test_graph_cache.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_graph_cache(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "test_graph_cache")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-fsanitize=address,undefined", "-I",
                        os.path.join(ROOT, "gpumatting_b200", "csrc"),
                        os.path.join(ROOT, "tests", "c", "test_graph_cache.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "Test PASSED" in r.stdout, r.stdout + r.stderr

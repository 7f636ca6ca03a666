"""The host-side work plans of the stages (tests/cpp/plan_checks.cpp, compiled
against the library)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIBDIR = os.path.join(ROOT, "enzo-e_gb300")
CUDA = "/usr/local/cuda"


@pytest.fixture(scope="module")
def checks(tmp_path_factory):
    if not os.path.exists(os.path.join(LIBDIR, "libmhdvlct_gb300.so")):
        pytest.skip("library not built")
    exe = str(tmp_path_factory.mktemp("plans") / "plan_checks")
    subprocess.run(
        ["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "include"),
         "-I", os.path.join(LIBDIR, "csrc"), "-I", os.path.join(CUDA, "include"),
         os.path.join(ROOT, "tests", "cpp", "plan_checks.cpp"), "-o", exe,
         "-L", LIBDIR, "-lmhdvlct_gb300", "-L", os.path.join(CUDA, "lib64"), "-lcudart",
         "-Wl,-rpath," + LIBDIR, "-Wl,-rpath," + os.path.join(CUDA, "lib64")],
        check=True, capture_output=True, text=True)
    return exe


@pytest.mark.parametrize("check", ["f64_tiles", "search", "search_time", "slabs"])
def test_plan(checks, check):
    r = subprocess.run([checks, check], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr

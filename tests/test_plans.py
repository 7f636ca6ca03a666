"""The host-side work plans of the stages (tests/cpp/plan_checks.cpp, compiled
against the library), and FP64 batches without room for the split stages'
workspace (tests/cpp/memory_checks.cpp, on a GPU)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIBDIR = os.path.join(ROOT, "enzo-e_gb300")
CUDA = "/usr/local/cuda"


def _build(name, tmp, *flags):
    if not os.path.exists(os.path.join(LIBDIR, "libmhdvlct_gb300.so")):
        pytest.skip("library not built")
    exe = str(tmp / name)
    subprocess.run(
        ["g++", "-std=c++17", "-O2", *flags, "-I", os.path.join(ROOT, "include"),
         "-I", os.path.join(LIBDIR, "csrc"), "-I", os.path.join(CUDA, "include"),
         os.path.join(ROOT, "tests", "cpp", name + ".cpp"), "-o", exe,
         "-L", LIBDIR, "-lmhdvlct_gb300", "-L", os.path.join(CUDA, "lib64"), "-lcudart", "-ldl",
         "-Wl,-rpath," + LIBDIR, "-Wl,-rpath," + os.path.join(CUDA, "lib64")],
        check=True, capture_output=True, text=True)
    return exe


@pytest.fixture(scope="module")
def checks(tmp_path_factory):
    return _build("plan_checks", tmp_path_factory.mktemp("plans"))


@pytest.mark.parametrize("check", ["f64_tiles", "search", "search_time", "slabs", "chunks"])
def test_plan(checks, check):
    r = subprocess.run([checks, check], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
def test_batches_without_room_for_the_workspace(tmp_path):
    # the program's own cudaMalloc stands before the runtime's
    exe = _build("memory_checks", tmp_path, "-rdynamic")
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr

"""The slab heap behind vectors and matrices (handle_heap.cuh) is host code:
random allocations and frees, with slabs that touch and slabs that do not."""
import os
import subprocess

from tests.conftest import ROOT


def test_blocks_stay_apart_and_everything_comes_back(tmp_path):
    exe = tmp_path / "handle_heap"
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "raptor_b200", "csrc"),
                           os.path.join(ROOT, "tests", "cxx", "handle_heap.cpp"), "-o", str(exe)])
    assert subprocess.run([str(exe)], capture_output=True, text=True, timeout=120).stdout == "ok\n"

"""The branch-and-bound heap filled with one value at once must be the heap
that pushing the keys one by one gives (tests/template_harness/heap_fill.cpp)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fill") / "heap_fill")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "product-graph-cycles_b200", "csrc"), "-o", exe,
                    os.path.join(HERE, "template_harness", "heap_fill.cpp")], check=True)
    return exe


@pytest.mark.parametrize("capacity", [1, 2, 7, 64, 333])
def test_fill_equals_pushes(harness, capacity):
    r = subprocess.run([harness, str(capacity), str(capacity)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout

"""Where a layer's entries lie in the streams of the other slot order, without a
GPU (tests/template_harness/positions.cpp)."""
import os
import subprocess

import numpy as np
import pytest

from cyclic_product_graphs import synthetic

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "product-graph-cycles_b200", "csrc")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("positions") / "positions")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "template_harness", "positions.cpp"),
                    os.path.join(CSRC, "graph_template.cpp")], check=True)
    return exe


@pytest.mark.parametrize("conj,prune", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("n,ny", [(33, 2), (90, 5), (301, 3)])
def test_entries_find_their_edge(harness, tmp_path, n, ny, conj, prune):
    EX = synthetic.directed_edges(synthetic.fibonacci_sphere(n)[1])
    EX = np.random.default_rng(n).permutation(n)[EX]  # ids that do not follow the mesh
    np.ascontiguousarray(EX.astype(np.int32)).tofile(tmp_path / "EX.bin")
    r = subprocess.run([harness, str(tmp_path / "EX.bin"), str(n), str(conj), str(prune), str(ny)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout

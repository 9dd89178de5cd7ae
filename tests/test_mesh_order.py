"""The mesh-ordered layer template (list slots along the mesh instead of by
node id) and the slice ranges of teams on local tables, without a GPU: a
harness (tests/template_harness/mesh.cpp) compares every node's in-edge list
with the template ordered by node ids, and the ranges with an exact search."""
import os
import subprocess

import numpy as np
import pytest

from cyclic_product_graphs import synthetic

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("mesh") / "mesh")
    csrc = os.path.join(ROOT, "product-graph-cycles_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", csrc, "-o", exe,
                    os.path.join(HERE, "template_harness", "mesh.cpp"),
                    os.path.join(csrc, "graph_template.cpp")], check=True)
    return exe


def _edges(kind):
    if kind == "tetrahedron":
        und = [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]
        return np.array(sorted(und + [(b, a) for a, b in und]), dtype=np.int32), 4
    n = int(kind)
    V, F = synthetic.fibonacci_sphere(n)
    EX = synthetic.directed_edges(F)
    if n == 90:  # edges in any order, two components, one direction missing here and there
        rng = np.random.default_rng(5)
        EX = np.concatenate([EX, EX + n])
        keep = rng.permutation(len(EX))[: len(EX) - 7]
        n = 2 * n
        assert len(np.unique(EX[keep])) == n
        EX = EX[keep]
    return np.ascontiguousarray(EX.astype(np.int32)), n


@pytest.mark.parametrize("conj,prune", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("kind", ["tetrahedron", "33", "90", "300"])
def test_mesh_order_keeps_every_list(harness, tmp_path, kind, conj, prune):
    EX, nv = _edges(kind)
    EX.tofile(tmp_path / "EX.bin")
    r = subprocess.run([harness, str(tmp_path / "EX.bin"), str(nv), str(conj), str(prune), "5"], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stdout

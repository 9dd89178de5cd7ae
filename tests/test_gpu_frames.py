"""SO(3) distances of frames whose normal and edge come close to parallel, on
either side of the angle (1e-4) below which the aligning rotation is taken from
an eigenvector instead of the frames' own directions, against the oracle's
singular value decomposition.

Bound, in radians.  A frame's third row is the cross product of edge and
normal, off by at most 4 eps / angle in direction; the aligning rotation moves
by no more than that (the singular values' pairwise sums are at least 1), twice
per distance and on both sides: 16 eps / 1e-6 = 3.6e-9 at the smallest angle
here.  A distance is 2 acos(ip), and four roundings of ip next to 1 are
2 sqrt(2 * 4 * eps / 2) = 6e-8.  Together below 1e-7."""
import numpy as np
import pytest

from cyclic_product_graphs import synthetic

pytestmark = pytest.mark.gpu

ANGLES = [np.pi / 2, 1.0, 2.0, 1e-2, np.pi - 1e-2, 2e-4, np.pi - 2e-4, 1.001e-4, 0.999e-4, np.pi - 0.999e-4,
          np.pi - 1.001e-4, 1e-6]


@pytest.mark.parametrize("prune", [False, True])
@pytest.mark.parametrize("order", [1, -1, 5])
def test_frames_near_parallel(cpg, oracle, prune, order):
    n = len(ANGLES)
    p = synthetic.make_pair(n_vertices=60, n_curve=n, feat_dim=8, seed=8)
    edge = p["VY"][p["EY"][:, 1]] - p["VY"][p["EY"][:, 0]]
    edge /= np.linalg.norm(edge, axis=1, keepdims=True)
    across = np.cross(edge, np.random.default_rng(3).standard_normal((n, 3)))
    across /= np.linalg.norm(across, axis=1, keepdims=True)
    angle = np.array([ANGLES[(i * order) % n] for i in range(n)])[:, None]
    NY = np.empty((n, 3))
    NY[p["EY"][:, 0]] = np.cos(angle) * edge + np.sin(angle) * across
    both = []
    for make in (cpg.product_graph_generator, oracle.OracleGenerator):
        g = make(p["VX"], p["EX"], p["VY"], p["EY"], p["feat_diff"], True, True, prune)
        g.set_normals(p["NX"], NY)
        g.set_cost_time_ratio_mode("plainso3", "feature")
        g.generate()
        both.append(g.get_cost_vector())
    assert both[0].shape == both[1].shape and np.isfinite(both[1]).all()
    assert both[1][:, 0].max() > 1.0  # distances of all sizes
    np.testing.assert_allclose(both[0][:, 0], both[1][:, 0], rtol=0, atol=1e-7)
    np.testing.assert_array_equal(both[0][:, 1], both[1][:, 1])

"""Conjugate energies with one row a thread or two (pruned, with frames, from
148 two-row work items on) against the oracle, either side of that line."""
import numpy as np
import pytest

from cyclic_product_graphs import synthetic

pytestmark = pytest.mark.gpu


# pruned: 142 work items, 168, 226 and 339, one and two layers past a chunk
@pytest.mark.parametrize("nv,ny,prune,reg", [(500, 30, True, True), (600, 30, True, True), (800, 31, True, True),
                                             (800, 32, True, True), (800, 33, True, True), (800, 33, True, False),
                                             (150, 33, False, True), (33, 16, True, True)])
@pytest.mark.parametrize("cost,time", [("robustso3", "feature"), ("vanilla", "lengthnormalisation")])
def test_rows_per_thread(cpg, oracle, nv, ny, prune, reg, cost, time):
    p = synthetic.make_pair(n_vertices=nv, n_curve=ny, feat_dim=4, seed=nv + ny)
    both = []
    for make in (cpg.product_graph_generator, oracle.OracleGenerator):
        g = make(p["VX"], p["EX"], p["VY"], p["EY"], p["feat_diff"], True, reg, prune)
        g.set_normals(p["NX"], p["NY"])
        g.set_cost_time_ratio_mode(cost, time)
        g.generate()
        both.append(g.get_cost_vector())
    # distances next to zero: four roundings of their cosine, 2 sqrt(4 eps) = 6e-8, and the loss's slope is below 1 there
    np.testing.assert_allclose(both[0], both[1], rtol=1e-9, atol=1e-7 if reg else 1e-9)
    assert np.array_equal(np.isnan(both[0]), np.isnan(both[1]))

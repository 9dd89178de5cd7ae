"""Plain energies with chunks of two, four and sixteen layers a thread, on both
sides of the lines between them (151,552 and 2,424,832 entries), against the
oracle bit for bit."""
import numpy as np
import pytest

from cyclic_product_graphs import synthetic

pytestmark = pytest.mark.gpu


# entries: 832 * 9, 832 * 2, 151k and 156k, 2.36 M and 2.48 M (layers that are no multiple of the chunk)
@pytest.mark.parametrize("nv,ny", [(42, 8), (42, 2), (300, 35), (300, 36), (2000, 89), (2000, 94)])
@pytest.mark.parametrize("reg,cost,time", [(False, "vanilla", "nomode"), (True, "feature", "lengthnormalisation")])
def test_plain_energy(cpg, oracle, nv, ny, reg, cost, time):
    p = synthetic.make_pair(n_vertices=nv, n_curve=ny, feat_dim=4, seed=nv + ny, with_normals=False)
    args = (p["VX"], p["EX"], p["VY"], p["EY"], p["feat_diff"], False, reg, False)
    both = []
    for make in (cpg.product_graph_generator, oracle.OracleGenerator):
        g = make(*args)
        g.set_cost_time_ratio_mode(cost, time)
        g.generate()
        both.append(g.get_cost_vector())
    assert np.array_equal(both[0], both[1])

"""What a new handle pays for its first cost matrix: no launch that a later one
does not make (the solvers' row masks wait for a solve), and the solves that
follow find what they need."""
import numpy as np
import pytest

from cyclic_product_graphs import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("conj", [False, True])
def test_first_costs_launch_what_later_ones_do(cpg, oracle, conj):
    p = synthetic.make_pair(n_vertices=70, n_curve=6, feat_dim=8, seed=2)
    args = (p["VX"], p["EX"], p["VY"], p["EY"], p["feat_diff"], conj, False, False)
    g, o = cpg.product_graph_generator(*args), oracle.OracleGenerator(*args)
    for h in (g, o):
        if conj:
            h.set_normals(p["NX"], p["NY"])
        h.set_cost_time_ratio_mode("vanilla", "lengthnormalisation" if conj else "nomode")
    counts = []
    for _ in range(2):
        n0 = cpg.kernel_launches()
        g.generate()
        costs = g.get_cost_vector()
        counts.append(cpg.kernel_launches() - n0)
    assert counts[0] == counts[1], counts
    assert np.array_equal(costs, o.get_cost_vector())
    got, want = g.solve_with_minimum_cost("dijkstragpu", 3), o.solve_with_minimum_cost("dijkstracpu", 3)
    assert got[0] == want[0] and got[1] == want[1] and np.array_equal(got[2], want[2])
    got, want = g.solve_with_cost_time_ratio("lawlergpu", 3), o.solve_with_cost_time_ratio("lawlercpu", 3)
    assert got[0] == want[0] and got[1] == want[1] and np.array_equal(got[2], want[2])

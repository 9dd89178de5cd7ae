"""Local tables beside which the two step buffers do not fit: the streams are
read in place.  A pruned conjugate graph of one CTA, 2,844 nodes a layer: about
110 KB of tables, 98 KB for each buffer of a step's costs and times."""
import numpy as np
import pytest

from cyclic_product_graphs import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,ny", [(2, 6), (4, 8)])
def test_streams_in_place(cpg, oracle, monkeypatch, K, ny):
    p = synthetic.make_pair(n_vertices=160, n_curve=ny, feat_dim=8, seed=K)
    args = (p["VX"], p["EX"], p["VY"], p["EY"], p["feat_diff"], True, False, True)
    g, o = cpg.product_graph_generator(*args), oracle.OracleGenerator(*args)
    for h in (g, o):
        h.set_normals(p["NX"], p["NY"])
        h.set_cost_time_ratio_mode("vanilla", "lengthnormalisation")
        h.generate()
    want = [o.solve_with_cost_time_ratio("lawlercpu", K)]
    got = [cpg.solve_batch([g], "lawlergpu", K, ctas_per_graph=1)[0]]
    # tables alone: less than the two buffers of 4-byte costs and times
    assert 0 < cpg.last_batch_profile()["smem_bytes"] < 2 * 8 * g.graph_info()["inter_slots_per_layer"]
    assert g.last_profile()["steps"] == g.last_stats()["sweeps"] * ny  # local tables, one depth
    monkeypatch.setenv("PGC_BF_BLOCKS", "1")
    want.append(o.solve_with_minimum_cost("dijkstracpu", K))
    got.append(g.solve_with_minimum_cost("dijkstragpu", K))
    g.generate()
    o.generate()
    want.append(o.solve_with_cost_time_ratio("lawlercpu", K))
    got.append(g.solve_with_cost_time_ratio("lawlergpu", K))
    for x, w in zip(got, want):
        assert x[0] == w[0] and x[1] == w[1] and np.array_equal(x[2], w[2])

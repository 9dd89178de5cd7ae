"""The profile's step count is the number of steps that ran: layers x depths a
sweep on local tables (the closing layer has its interlayer step only), one
depth where layers have no intralayer edges, and every layer's depths in global
memory."""
import pytest

from cyclic_product_graphs import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("local", ["1", "0"])
@pytest.mark.parametrize("conj,prune,K,ny", [(False, False, 1, 5), (False, False, 4, 6), (True, False, 3, 5),
                                             (True, True, 4, 6)])
def test_steps_per_sweep(cpg, monkeypatch, local, conj, prune, K, ny):
    monkeypatch.setenv("PGC_BF_LOCAL", local)
    p = synthetic.make_pair(n_vertices=70, n_curve=ny, feat_dim=8, seed=5)
    g = cpg.product_graph_generator(p["VX"], p["EX"], p["VY"], p["EY"], p["feat_diff"], conj, False, prune)
    if conj:
        g.set_normals(p["NX"], p["NY"])
    g.set_cost_time_ratio_mode("vanilla", "lengthnormalisation" if conj else "nomode")
    depths = 1 if prune else K
    want = ny * depths if local == "1" else (ny + 1) * depths - 1
    cpg.solve_batch([g], "lawlergpu", K, regenerate=True)
    assert g.last_profile()["steps"] == g.last_stats()["sweeps"] * want > 0
    for solve in (g.solve_with_cost_time_ratio, g.solve_with_minimum_cost):
        solve("lawlergpu" if solve == g.solve_with_cost_time_ratio else "dijkstragpu", K)
        assert g.last_profile()["steps"] == g.last_stats()["sweeps"] * want > 0

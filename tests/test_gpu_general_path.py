"""Sweeps on records in global memory, which serve every graph whose tables do
not fit its team's shared memory: reached here by the team's size, in single
solves and in a batch, against the oracle; and a team's ranges and wait lists,
which a repeated solve finds as the first one left them."""
import ctypes

import numpy as np
import pytest

from cyclic_product_graphs import synthetic

pytestmark = pytest.mark.gpu


def _handles(cpg, oracle, p, conj, modes):
    args = (p["VX"], p["EX"], p["VY"], p["EY"], p["feat_diff"], conj, False, False)
    g, o = cpg.product_graph_generator(*args), oracle.OracleGenerator(*args)
    for h in (g, o):
        if conj:
            h.set_normals(p["NX"], p["NY"])
        h.set_cost_time_ratio_mode(*modes)
    return g, o


def _same(got, want):
    assert got[0] == want[0] and got[1] == want[1], (got[:2], want[:2])
    assert np.array_equal(got[2], want[2])


def _uploads(cpg):
    n = ctypes.c_int64()
    assert cpg._lib.pgc_team_uploads(ctypes.byref(n)) == 0
    return n.value


# 600 vertices: 10,764 nodes a layer, about 390 KB of tables for each of two CTAs
@pytest.mark.parametrize("blocks", ["1", "2", "0"])
def test_tables_that_do_not_fit(cpg, oracle, monkeypatch, blocks):
    monkeypatch.setenv("PGC_BF_BLOCKS", blocks)
    p = synthetic.make_pair(n_vertices=600, n_curve=9, feat_dim=8, seed=3)
    g, o = _handles(cpg, oracle, p, True, ("vanilla", "lengthnormalisation"))
    for _ in range(2):
        g.generate()
        o.generate()
        _same(g.solve_with_cost_time_ratio("lawlergpu", 3), o.solve_with_cost_time_ratio("lawlercpu", 3))
        _same(g.solve_with_minimum_cost("dijkstragpu", 3), o.solve_with_minimum_cost("dijkstracpu", 3))


@pytest.mark.parametrize("blocks", ["2", "0"])
@pytest.mark.parametrize("solve", ["ratio", "cost"])
def test_a_repeated_solve_uploads_no_team(cpg, oracle, monkeypatch, blocks, solve):
    monkeypatch.setenv("PGC_BF_BLOCKS", blocks)
    p = synthetic.make_pair(n_vertices=600, n_curve=9, feat_dim=8, seed=3)
    g, _ = _handles(cpg, oracle, p, True, ("vanilla", "lengthnormalisation"))
    for i in range(3):
        g.generate()
        before = _uploads(cpg)
        if solve == "ratio":
            g.solve_with_cost_time_ratio("lawlergpu", 3)
        else:
            g.solve_with_minimum_cost("dijkstragpu", 3)
        assert _uploads(cpg) - before <= (2 if i == 0 else 0)


def test_batch_with_a_graph_that_does_not_fit(cpg, oracle):
    sizes = [(600, 3), (40, 3), (80, 2)]
    pairs = [_handles(cpg, oracle, synthetic.make_pair(n_vertices=n, n_curve=7, feat_dim=8, seed=n), True,
                      ("vanilla", "lengthnormalisation")) for n, _ in sizes]
    for (g, o), (_, K) in zip(pairs, sizes):
        g.set_max_depth_cost_time_ratio(K)
    want = [o.solve_with_cost_time_ratio("lawlercpu", K) for (_, o), (_, K) in zip(pairs, sizes)]
    for team in (1, 2):
        got = cpg.solve_batch([g for g, _ in pairs], "lawlergpu", ctas_per_graph=team, regenerate=True)
        for x, w in zip(got, want):
            _same(x, w)


def _shuffled(p, seed):
    """The pair with its X vertices renumbered at random."""
    at = np.random.default_rng(seed).permutation(len(p["VX"]))  # new id of an old vertex
    q = dict(p)
    q["VX"], q["feat_diff"] = np.empty_like(p["VX"]), np.empty_like(p["feat_diff"])
    q["VX"][at], q["feat_diff"][at] = p["VX"], p["feat_diff"]
    q["EX"] = np.ascontiguousarray(at[p["EX"]].astype(p["EX"].dtype))
    return q


# lists by node id: more depths than tables hold, two layers, one CTA and several, ids that follow the mesh and not,
# streams of floats and of doubles
@pytest.mark.parametrize("K,ny", [(5, 9), (6, 4), (2, 2), (5, 2)])
@pytest.mark.parametrize("blocks", ["0", "3"])
@pytest.mark.parametrize("shuffle,wide", [(False, False), (True, False), (True, True)])
def test_plain_lists_by_node(cpg, oracle, monkeypatch, K, ny, blocks, shuffle, wide):
    monkeypatch.setenv("PGC_BF_BLOCKS", blocks)
    p = synthetic.make_pair(n_vertices=150, n_curve=ny, feat_dim=8, seed=K + ny, with_normals=False)
    if shuffle:
        p = _shuffled(p, K)
    g, o = _handles(cpg, oracle, p, False, ("feature", "lengthnormalisation"))
    for _ in range(2):
        if wide:  # past float's integers after the rescale
            c = np.random.default_rng(ny).uniform(1.0, 2.0, size=g.get_cost_vector().shape) * [[1e6, 1.0]]
            g.set_cost_vector(c)
            o.set_cost_vector(c)
        else:
            g.generate()
            o.generate()
        _same(g.solve_with_minimum_cost("dijkstragpu", K), o.solve_with_minimum_cost("dijkstracpu", K))
        _same(g.solve_with_cost_time_ratio("lawlergpu", K), o.solve_with_cost_time_ratio("lawlercpu", K))


def test_plain_lists_by_node_in_a_batch(cpg, oracle):
    sizes = [(150, 5, 7), (97, 2, 5), (333, 6, 4)]
    pairs = [_handles(cpg, oracle, _shuffled(synthetic.make_pair(n_vertices=n, n_curve=ny, feat_dim=8, seed=n), n),
                      False, ("vanilla", "nomode")) for n, _, ny in sizes]
    for (g, _), (_, K, _) in zip(pairs, sizes):
        g.set_max_depth_cost_time_ratio(K)
    want = [o.solve_with_cost_time_ratio("lawlercpu", K) for (_, o), (_, K, _) in zip(pairs, sizes)]
    for team in (1, 4):
        got = cpg.solve_batch([g for g, _ in pairs], "lawlergpu", ctas_per_graph=team, regenerate=True)
        for x, w in zip(got, want):
            _same(x, w)

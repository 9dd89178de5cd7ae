"""A wait for a staged copy that runs out (PGC_BF_TEST_STALL_COPY names the CTA
whose steps give their copies no poll): the solve ends promptly with
PGC_ERR_TIMEOUT once the copies have landed after all, on local tables and on
records in global memory, with one CTA and with several; graphs that follow in
the same launch find no copy in their tables; and the same handles then solve
as the oracle does.  Nothing faults: the copies land, only the wait gives up."""
import time

import numpy as np
import pytest

from cyclic_product_graphs import synthetic

pytestmark = pytest.mark.gpu

PGC_ERR_TIMEOUT = -7


def _pair(seed, n=642):
    p = synthetic.make_pair(n_vertices=n, n_curve=20, feat_dim=8, seed=seed)
    return p["VX"], p["EX"], p["VY"], p["EY"], p["feat_diff"], False, False, False


def _same(got, want):
    assert got[0] == want[0] and got[1] == want[1], (got[:2], want[:2])
    assert np.array_equal(got[2], want[2])


@pytest.mark.parametrize("local", ["1", "0"])
@pytest.mark.parametrize("blocks,cta", [("1", "0"), ("8", "0"), ("8", "5")])
def test_stalled_copy_ends_the_solve(cpg, oracle, monkeypatch, local, blocks, cta):
    args = _pair(4)
    g, o = cpg.product_graph_generator(*args), oracle.OracleGenerator(*args)
    monkeypatch.setenv("PGC_BF_LOCAL", local)
    monkeypatch.setenv("PGC_BF_BLOCKS", blocks)
    monkeypatch.setenv("PGC_BF_THREADS", "64")  # two warps a CTA: CTA 5 of 8 has slices in both layouts
    monkeypatch.setenv("PGC_BF_TEST_STALL_COPY", cta)
    for solve, name in ((g.solve_with_cost_time_ratio, "lawlergpu"), (g.solve_with_minimum_cost, "dijkstragpu")):
        t0 = time.perf_counter()
        with pytest.raises(cpg.PGCError) as e:
            solve(name, 2)
        assert e.value.code == PGC_ERR_TIMEOUT and "ran out" in str(e.value)
        assert time.perf_counter() - t0 < 10.0
    monkeypatch.delenv("PGC_BF_TEST_STALL_COPY")
    g.generate()
    _same(g.solve_with_cost_time_ratio("lawlergpu", 2), o.solve_with_cost_time_ratio("lawlercpu", 2))
    _same(g.solve_with_minimum_cost("dijkstragpu", 2), o.solve_with_minimum_cost("dijkstracpu", 2))


@pytest.mark.parametrize("local", ["1", "0"])
@pytest.mark.parametrize("team", [1, 4])
def test_stalled_copies_in_a_batch(cpg, monkeypatch, local, team):
    monkeypatch.setenv("PGC_BF_LOCAL", local)
    gens = [cpg.product_graph_generator(*_pair(10 + i, 200 + 37 * i)) for i in range(5)]
    want = cpg.solve_batch(gens, "lawlergpu", 2, ctas_per_graph=team, regenerate=True)
    monkeypatch.setenv("PGC_BF_TEST_STALL_COPY", "0")
    with pytest.raises(cpg.PGCError) as e:
        cpg.solve_batch(gens, "lawlergpu", 2, ctas_per_graph=team, regenerate=True)
    assert e.value.code == PGC_ERR_TIMEOUT
    monkeypatch.delenv("PGC_BF_TEST_STALL_COPY")
    for got, w in zip(cpg.solve_batch(gens, "lawlergpu", 2, ctas_per_graph=team, regenerate=True), want):
        _same(got, w)


def test_stall_hook_outside_the_team_changes_nothing(cpg, oracle, monkeypatch):
    args = _pair(6, 162)
    g, o = cpg.product_graph_generator(*args), oracle.OracleGenerator(*args)
    monkeypatch.setenv("PGC_BF_BLOCKS", "4")
    monkeypatch.setenv("PGC_BF_TEST_STALL_COPY", "99")
    _same(g.solve_with_cost_time_ratio("lawlergpu", 2), o.solve_with_cost_time_ratio("lawlercpu", 2))

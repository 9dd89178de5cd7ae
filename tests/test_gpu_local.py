"""Sweeps on per-CTA local tables against the sweeps in global memory
(PGC_BF_LOCAL=0), bit for bit: the answers, the cycle's edges, and how often
the solver swept and branched.  Team sizes from one CTA to more CTAs than a
slice each, odd and even layer counts, every depth the tables hold, costs that
are exact floats and costs that are not (double streams), and costs with
infinities and NaN."""
import numpy as np
import pytest

from cyclic_product_graphs import synthetic

pytestmark = pytest.mark.gpu

SOLVES = (("ratio", "lawlergpu"), ("cost", "dijkstragpu"))


def _solve(g, kind, name, K):
    try:
        r = g.solve_with_cost_time_ratio(name, K) if kind == "ratio" else g.solve_with_minimum_cost(name, K)
    except RuntimeError as e:
        return ("error", str(e))
    st = g.last_stats()
    return (r[0], np.float32(r[1]).tobytes(), r[2].tobytes(), g.last_cycle_edges().tobytes(), st["sweeps"],
            st["branches"], st["bf_calls"])


def _both(cpg, monkeypatch, make, K, costs=None):
    out = []
    for local in ("1", "0"):
        monkeypatch.setenv("PGC_BF_LOCAL", local)
        g = make()
        got = []
        for kind, name in SOLVES:
            if costs is None:
                g.generate()
            else:
                g.set_cost_vector(costs)
            got.append(_solve(g, kind, name, K))
        out.append(got)
    assert out[0] == out[1]
    return out[0]


def _maker(cpg, p, conj=False, prune=False, cost="vanilla", time="nomode"):
    def make():
        g = cpg.product_graph_generator(p["VX"], p["EX"], p["VY"], p["EY"], p["feat_diff"], conj, False, prune)
        if conj:
            g.set_normals(p["NX"], p["NY"])
        g.set_cost_time_ratio_mode(cost, time)
        return g
    return make


@pytest.mark.parametrize("blocks", ["0", "1", "2", "7", "32"])
@pytest.mark.parametrize("K,ny", [(1, 9), (2, 3), (2, 14), (3, 9), (4, 6), (4, 7)])
def test_plain(cpg, monkeypatch, blocks, K, ny):
    monkeypatch.setenv("PGC_BF_BLOCKS", blocks)
    p = synthetic.make_pair(n_vertices=270, n_curve=ny, feat_dim=8, seed=K * 100 + ny)
    _both(cpg, monkeypatch, _maker(cpg, p, cost="feature", time="lengthnormalisation"), K)


@pytest.mark.parametrize("blocks", ["0", "1", "5", "40"])
@pytest.mark.parametrize("K,ny,prune", [(2, 8, False), (3, 7, False), (4, 4, False), (3, 8, True), (4, 5, True)])
def test_conjugate(cpg, monkeypatch, blocks, K, ny, prune):
    monkeypatch.setenv("PGC_BF_BLOCKS", blocks)
    p = synthetic.make_pair(n_vertices=90, n_curve=ny, feat_dim=8, seed=K * 100 + ny)
    _both(cpg, monkeypatch, _maker(cpg, p, conj=True, prune=prune, cost="vanilla", time="lengthnormalisation"), K)


@pytest.mark.parametrize("blocks", ["1", "6"])
@pytest.mark.parametrize("K,ny", [(2, 6), (3, 5)])
@pytest.mark.parametrize("kind", ["wide", "infinite", "nan", "ties"])
def test_unusual_costs(cpg, monkeypatch, blocks, K, ny, kind):
    monkeypatch.setenv("PGC_BF_BLOCKS", blocks)
    p = synthetic.make_pair(n_vertices=100, n_curve=ny, feat_dim=8, seed=7)
    make = _maker(cpg, p)
    rows = make().get_cost_vector().shape[0]
    rng = np.random.default_rng(K)
    c = rng.uniform(0.5, 2.0, size=(rows, 1 if K == 2 else 2))
    if kind == "wide":  # the rescale clips, and the minimum cost keeps them as they are
        c[:, 0] *= 10.0 ** rng.integers(-3, 9, size=rows)
    elif kind == "infinite":
        c[rng.integers(0, rows, size=rows // 20), 0] = np.inf
    elif kind == "nan":
        c[rng.integers(0, rows, size=rows // 50), 0] = np.nan
    else:
        c = rng.integers(1, 4, size=c.shape).astype(np.float64)
    _both(cpg, monkeypatch, make, K, costs=c)


def test_batched_mixed_sizes(cpg, monkeypatch):
    """Graphs whose tables fit a batch team and one whose depths do not."""
    pairs = [synthetic.make_pair(n_vertices=n, n_curve=m, feat_dim=8, seed=s)
             for n, m, s in ((100, 8, 1), (333, 11, 2), (700, 6, 3), (150, 9, 4))]
    res = []
    for local in ("1", "0"):
        monkeypatch.setenv("PGC_BF_LOCAL", local)
        gens = [_maker(cpg, p)() for p in pairs]
        for g, K in zip(gens, (1, 2, 3, 5)):
            g.set_max_depth_cost_time_ratio(K)
        for team in (0, 1, 4):
            r = cpg.solve_batch(gens, "lawlergpu", ctas_per_graph=team, regenerate=True)
            res.append([(x[0], x[1], x[2].tobytes()) for x in r])
    assert all(x == res[0] for x in res)

"""The largest feature difference, which the feature time is measured from,
found by the host (up to 20,480 entries) or on the device: either side of the
line, at the matrix's ends, and held twice."""
import numpy as np
import pytest

from cyclic_product_graphs import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [12, 204, 205, 240])  # 100 vertices: 20,400 and 20,500 entries
@pytest.mark.parametrize("where", ["first", "last", "twice"])
def test_largest_feature_difference(cpg, ny, where):
    nv = 100
    p = synthetic.make_pair(n_vertices=nv, n_curve=ny, feat_dim=4, seed=ny)
    fd = np.array(p["feat_diff"], dtype=np.float64)
    flat = fd.reshape(-1)
    top = 2.0 * flat.max()
    for at in {"first": [0], "last": [flat.size - 1], "twice": [flat.size // 3, flat.size // 2]}[where]:
        flat[at] = top
    g = cpg.product_graph_generator(p["VX"], p["EX"], p["VY"], p["EY"], fd, True, False, False)
    g.set_normals(p["NX"], p["NY"])
    g.set_cost_time_ratio_mode("plainso3", "feature")
    g.generate()
    times = g.get_cost_vector()[:, 1]
    top32 = float(np.float32(top))
    assert times.max() == max(0.0, top32 - flat.min()) and times.min() == max(0.0, top32 - top)

"""A team shape in the autotuner's cache belongs to the kernels it was timed
with: an entry of other kernels, or of none that it names, is timed again."""
import json

import pytest

from test_autotune_host import FakeGenerator


@pytest.mark.parametrize("edit", [lambda e: e.pop("kernels"), lambda e: e.update(kernels=e["kernels"] - 1),
                                  lambda e: e.update(kernels=None)])
def test_entry_of_other_kernels_is_timed_again(cpg, tmp_path, edit):
    cache = tmp_path / "c.json"
    cpg.autotune(FakeGenerator(times={(8, 320): 1.0}), 3, candidates=[(0, 0), (8, 320)], cache_path=str(cache))
    entries = json.loads(cache.read_text())
    (key,) = entries
    edit(entries[key])
    cache.write_text(json.dumps(entries))
    g = FakeGenerator(times={(16, 640): 1.0})
    e = cpg.autotune(g, 3, candidates=[(0, 0), (16, 640)], cache_path=str(cache))
    assert not e["cached"] and g.solves == 4 and g.shape == (16, 640)
    assert json.loads(cache.read_text())[key]["ctas"] == 16
    again = FakeGenerator()
    assert cpg.autotune(again, 3, cache_path=str(cache))["cached"] and again.solves == 0 and again.shape == (16, 640)

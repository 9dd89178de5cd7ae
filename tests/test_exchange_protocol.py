"""The rule by which CTAs on local tables report and wait (local_sweep in
csrc/bf_local.cuh), restated and run in random orders without a GPU: no team
comes to a stand, over several sweeps, and no record is overwritten before
every neighbour has read the one before it."""
import random

import pytest


def _sweeps(depths, layers, sweeps):
    out, step = [], 0
    for s in range(sweeps):
        for l in range(0 if depths > 1 else 1, layers + 1):
            for k in range(1 if l == 0 else 0, 1 if l == layers else depths):
                step += 1
                out.append((s, l, k, step))
    return out


def _run(depths, layers, ctas, seed, closing_report=True):
    rng = random.Random(seed)
    near = {c: [d for d in (c - 1, c + 1) if 0 <= d < ctas] for c in range(ctas)}
    steps = _sweeps(depths, layers, 3)
    where = {(s, l, k): i for i, (s, l, k, _) in enumerate(steps)}
    done, pos, relaxed = [0] * ctas, [0] * ctas, [-1] * ctas
    idle = 0
    while min(pos) < len(steps):
        if idle > 200 * ctas:
            return False
        idle += 1
        c = rng.randrange(ctas)
        if pos[c] == len(steps):
            continue
        s, l, k, step = steps[pos[c]]
        if relaxed[c] < pos[c]:
            if pos[c] and steps[pos[c] - 1][0] != s and min(pos) < pos[c]:
                continue  # the barrier between sweeps
            # the step's records replace those of two layers before, which the
            # neighbours read at the end of that step
            before = where.get((s, l - 2, k))
            assert before is None or all(pos[d] > before for d in near[c]), (depths, layers, ctas, seed)
            relaxed[c] = pos[c]
        else:
            if l < layers and any(relaxed[d] < pos[c] for d in near[c]):
                continue  # halo records not there yet
            if l < layers and k + 1 == depths and any(done[d] < step - depths for d in near[c]):
                continue  # a neighbour has not finished the layer before
            if closing_report if l == layers else k + 1 == depths:
                done[c] = step
            pos[c] += 1
        idle = 0
    return True


@pytest.mark.parametrize("depths", [1, 2, 3, 4])
@pytest.mark.parametrize("layers", [3, 4, 7])
def test_no_stand_and_no_early_overwrite(depths, layers):
    for ctas in (2, 3, 6):
        for seed in range(5):
            assert _run(depths, layers, ctas, seed)


def test_one_depth_needs_the_closing_layers_report():
    """Without it every CTA's first wait of the next sweep is for a report that
    only comes after it."""
    assert not _run(1, 4, 3, 0, closing_report=False)

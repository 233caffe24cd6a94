"""The dependent launches of a loop trial.

A trial's position update and gather start while the launch before them
drains, its bin adds where they take at most a block an SM (152), the field's
first pass up to 128 bins; all wait for that launch's results.  The batched
form's stages are ordinary launches of the same sums, so a batch of one gives
the same bits: at the last size of the bin adds' rule and the first beyond,
on both sides of the field's, with filler cells (two launches of bin adds in a
row), at a single block, in graphs and launched one by one.

The wirelength launches of one call wait for one another only at their ends (three of
the four up to 600k nets, all four beyond); one launch of the same nets gives
the same gradient bit for bit.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BLOCK_NODES = 2048  # the batched form's grid policy
LINE = 152 * BLOCK_NODES


@pytest.fixture(scope="module")
def ap():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aieplace_gb300 import build

    build.build()
    import aieplace_gb300

    return aieplace_gb300


@pytest.mark.parametrize("graph", [1, 0])
@pytest.mark.parametrize("cells,bins,fillers", [(200, 32, 0), (3000, 64, 1), (20_000, 128, 0), (LINE, 256, 0),
                                                (LINE + 1, 256, 0), (LINE - 1, 256, 1)])
def test_dependent_launches_match_ordinary_ones(ap, cells, bins, fillers, graph):
    nl = ap.synth.generate(dict(num_cells=cells, num_nets=cells, num_macros=0, num_pads=24, unit_cells=1, degree_mix=0,
                                locality=0.0, window=64, target_density=0.9,
                                die_side=float(math.ceil(math.sqrt(cells / 0.8))), bins=bins), seed=3)
    with ap.BatchPlacer([nl], filler_cells=fillers) as b:
        b.initialize_placement(seed=7, sigma=1.0)
        b.step(16)
        bx, by = b.positions(0)
        bs = b.stats(0)
    with ap.Placer(nl, block_nodes=BLOCK_NODES, filler_cells=fillers, use_graph=graph) as p:
        p.initialize_placement(seed=7, sigma=1.0)
        p.step_async(16)
        x, y = p.positions()
        s = p.stats()
    np.testing.assert_array_equal(bx, x)
    np.testing.assert_array_equal(by, y)
    assert bs["hpwl"] == s["hpwl"] and bs["overflow"] == s["overflow"]


@pytest.mark.parametrize("cells", [LINE, 2 * LINE])
def test_overlapping_wirelength_launches_match_one(ap, cells):
    nl = ap.synth.generate(dict(ap.synth.batch_specs(1, seed=1, lo=cells, hi=cells)[0], bins=512), seed=5)
    rng = np.random.default_rng(2)
    n = len(nl["node_w"])
    die = nl["die"]
    x = rng.uniform(0, die[2] * 0.99, n).astype(np.float32)
    y = rng.uniform(0, die[3] * 0.99, n).astype(np.float32)
    gamma = 2.0 * float(die[2]) / 512
    with ap.Placer(nl, bins=512, block_nodes=8192) as one, ap.Placer(nl, bins=512) as four:
        gx, gy, wa, hpwl = one.compute_all_partials(x, y, gamma)
        for _ in range(4):
            r = four.compute_all_partials(x, y, gamma)
            np.testing.assert_array_equal(r[0], gx)
            np.testing.assert_array_equal(r[1], gy)
            # FP32 sums of positive terms: at most 32 a thread and 8 levels of
            # a block's tree, each to 2^-24; compensated beyond
            assert abs(r[2] / wa - 1) < 2 * 40 * 2.0 ** -24 and abs(r[3] / hpwl - 1) < 2 * 40 * 2.0 ** -24

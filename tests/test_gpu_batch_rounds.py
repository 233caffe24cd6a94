"""The batched form's position update and gather in each of their occupancies: the
launch takes the one that runs its items (2048 nodes each here) in the fewest rounds
of resident blocks, 456, 608 or 760 of the update and 608 or 760 of the gather.  An
instance's results are its own launches' bit for bit in all of them.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ap():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aieplace_gb300 import build

    build.build()
    import aieplace_gb300

    return aieplace_gb300


def design(ap, cells):
    return ap.synth.generate(dict(num_cells=cells, num_nets=cells, num_macros=0, num_pads=8, unit_cells=1, degree_mix=0,
                                  locality=0.0, window=64, target_density=0.9,
                                  die_side=float(math.ceil(math.sqrt(cells / 0.8))), bins=32), seed=2)


@pytest.mark.parametrize("n,blocks", [(1, 1), (114, 4), (116, 4), (152, 4), (153, 4), (152, 5), (153, 5)])
def test_batch_matches_own_launches(ap, n, blocks):
    """items n * blocks: on both sides of 456, 608 and 760."""
    nl = design(ap, 2048 * (blocks - 1) + 100)
    with ap.BatchPlacer([nl] * n) as b:
        assert b.info()["form"] == "persistent"
        b.initialize_placement(seed=3, sigma=1.0)
        b.step(10)
        got = {i: (b.positions(i), b.stats(i)) for i in {0, n // 2, n - 1}}
    for i, ((x, y), s) in got.items():
        with ap.Placer(nl, block_nodes=2048) as p:
            p.initialize_placement(seed=3 + i, sigma=1.0)
            p.step_async(10)
            px, py = p.positions()
            ps = p.stats()
        np.testing.assert_array_equal(x, px)
        np.testing.assert_array_equal(y, py)
        assert s["hpwl"] == ps["hpwl"] and s["overflow"] == ps["overflow"] and s["alpha"] == ps["alpha"]

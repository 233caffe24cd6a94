"""The sums that end a loop trial: the overflow's partials of the field's first
pass, one block's (32 bins) to 1024 (4096 bins), folded with the gather's.

The overflow is a sum of whole numbers, so the loop's value equals that of a
placement initialised at the accepted positions, whose density kernel folds its
own sums.
"""
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


@pytest.mark.parametrize("cells,bins", [(200, 32), (3000, 64), (3000, 512), (3000, 1024), (3000, 2048), (300_000, 4096)])
def test_loop_overflow_equals_initial_evaluation(ap, cells, bins):
    spec = dict(ap.synth.batch_specs(1, seed=2, lo=cells, hi=cells)[0], bins=bins)
    nl = ap.synth.generate(spec, seed=9)
    assert nl["die"][0] == 0 and nl["die"][1] == 0  # positions read back are the loop's to the bit
    with ap.Placer(nl, bins=bins) as p, ap.Placer(nl, bins=bins) as q:
        p.initialize_placement(seed=5, sigma=1.0)
        p.perform_iteration(3)
        s = p.stats()
        assert s["iteration"] == 3
        q.initialize_placement(*p.positions())
        t = q.stats()
    assert (s["overflow"], s["overflow_abs"]) == (t["overflow"], t["overflow_abs"])

"""A handle's captured trials serve every placement after the one they were made
for: a handle that was placed, stepped and placed again goes on bit for bit like a
fresh one, in graphs of one trial and of four, whatever came between (a log, a
snapshot restored, a surrogate attached and taken off, another stream).
"""
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


CASES = {
    "c0_32": dict(preset="c0", bins=32),
    "small_128": dict(preset="c1_small", bins=128),
    "fillers_64": dict(preset="c1_small", bins=64, filler_cells=1),
    "mixed_256": dict(preset="c1_small", bins=256, field_solver="bf16x3"),
    "backtracks_128": dict(preset="c1_small", bins=128, max_backtracks=2),
}


def start(nl, seed):
    rng = np.random.default_rng(seed)
    x, y = nl["node_x"].copy(), nl["node_y"].copy()
    mov = nl["node_fixed"] == 0
    w, h = float(nl["die"][2]), float(nl["die"][3])
    x[mov] = rng.uniform(0.2 * w, 0.7 * w, mov.sum())
    y[mov] = rng.uniform(0.2 * h, 0.7 * h, mov.sum())
    return x, y


def go(pl, xy, n):
    pl.initialize_placement(*xy)
    pl.perform_iteration(n)
    return pl.positions(), pl.stats()


def same(a, b):
    (xa, ya), sa = a
    (xb, yb), sb = b
    np.testing.assert_array_equal(xa, xb)
    np.testing.assert_array_equal(ya, yb)
    assert sa == sb


def nothing(ap, pl, tmp_path):
    pass


def log(ap, pl, tmp_path):
    pl.set_log(str(tmp_path / "log"), capacity=4)
    pl.perform_iteration(6)


def restore(ap, pl, tmp_path):
    blob = pl.snapshot()
    pl.perform_iteration(5)
    pl.restore(blob)
    pl.perform_iteration(2)


def surrogate(ap, pl, tmp_path):
    with ap.Surrogate(factor=2, kernels=(3, 1, 1, 1)) as s:
        pl.attach_surrogate(s)
        pl.perform_iteration(5)
        pl.attach_surrogate(None)


def stream(ap, pl, tmp_path):
    import torch

    pl._stream = torch.cuda.Stream()  # kept alive with the handle
    pl.set_stream(pl._stream.cuda_stream)
    pl.perform_iteration(5)


@pytest.mark.parametrize("between", [nothing, log, restore, surrogate, stream], ids=lambda f: f.__name__)
@pytest.mark.parametrize("case", CASES)
def test_second_placement_matches_fresh_handle(ap, tmp_path, case, between):
    kw = dict(CASES[case])
    nl = ap.synth.generate(kw.pop("preset"), seed=4)
    if between is surrogate and kw["bins"] < 64:
        pytest.skip("the coarse grid of factor 2 would have 16 bins")
    a, b = start(nl, 1), start(nl, 2)
    steps = (11, 3)  # two graphs of four and three of one; one by one
    fresh = []
    for n in steps:
        with ap.Placer(nl, **kw) as pl:
            fresh.append(go(pl, b, n))
    with ap.Placer(nl, **kw) as pl:
        go(pl, a, 9)
        between(ap, pl, tmp_path)
        for n, want in zip(steps, fresh):
            same(go(pl, b, n), want)

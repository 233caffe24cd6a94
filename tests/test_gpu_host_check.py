"""Values that are not finite in host arrays, on both sides of the size up to which
the host looks for them (16384 nodes; beyond, a kernel sets a flag): the calls refuse
them and work on afterwards.  The initial placement looks at movable nodes only, the
stage calls at all.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AP_ERR_NONFINITE = 3


@pytest.fixture(scope="module")
def ap():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aieplace_gb300 import build

    build.build()
    import aieplace_gb300

    return aieplace_gb300


def design(ap, nodes):
    macros = 4
    nl = ap.synth.generate(dict(num_cells=nodes - macros, num_nets=nodes, num_macros=macros, num_pads=0, unit_cells=0,
                                degree_mix=1, locality=0.8, window=64, target_density=0.7, die_side=0.0, bins=64), seed=5)
    p = np.random.default_rng(6).permutation(nodes)  # the macros among the cells
    for k in ("node_w", "node_h", "node_x", "node_y", "node_fixed"):
        nl[k] = np.ascontiguousarray(nl[k][p])
    inv = np.empty_like(p)
    inv[p] = np.arange(nodes)
    nl["pin_node"] = inv[nl["pin_node"]].astype(np.int32)
    return nl


@pytest.mark.parametrize("nodes", [576, 16384, 16385, 16389])  # 4 of them fixed: initial placements of nodes - 4
def test_not_finite_is_refused(ap, nodes):
    nl = design(ap, nodes)
    movable, fixed = np.flatnonzero(nl["node_fixed"] == 0), np.flatnonzero(nl["node_fixed"])
    rng = np.random.default_rng(1)
    x, y = nl["node_x"].copy(), nl["node_y"].copy()
    for v in (x, y):
        v[movable] = rng.uniform(0, 0.9 * float(nl["die"][2]), len(movable))
    ex = rng.standard_normal(64 * 64).astype(np.float32)

    def with_value(v, at, value):
        w = v.copy()
        w[at] = value
        return w

    with ap.Placer(nl) as pl:
        stages = (lambda x, y: pl.compute_all_partials(x, y, 4.0), pl.compute_overlaps,
                  lambda x, y: pl.compute_node_forces(x, y, ex, ex, 4.0, 0.1))
        want = [f(x, y) for f in stages]
        pl.initialize_placement(x, y)
        pl.perform_iteration(2)
        before = pl.positions(), pl.stats()
        for value in (np.nan, np.inf, -np.inf):
            for at in (movable[0], movable[-1]):
                for xy in ((with_value(x, at, value), y), (x, with_value(y, at, value))):
                    for f in (*stages, pl.initialize_placement):
                        with pytest.raises(ap.APError) as e:
                            f(*xy)
                        assert e.value.status == AP_ERR_NONFINITE
            xf = with_value(x, fixed[-1], value)
            for f in stages:
                with pytest.raises(ap.APError) as e:
                    f(xf, y)
                assert e.value.status == AP_ERR_NONFINITE
        after = pl.positions(), pl.stats()
        np.testing.assert_array_equal(before[0], after[0])
        assert before[1] == after[1]
        for f, w in zip(stages, want):
            got = f(x, y)
            for u, v in zip(got, w) if isinstance(w, tuple) else ((got, w),):
                np.testing.assert_array_equal(u, v)
        pl.initialize_placement(with_value(x, fixed[0], np.nan), y)  # a fixed node's entry is not read
        pl.perform_iteration(2)
        after = pl.positions(), pl.stats()
        np.testing.assert_array_equal(before[0], after[0])
        assert before[1] == after[1]

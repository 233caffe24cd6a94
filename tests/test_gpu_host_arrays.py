"""Calls on host arrays in netlist order.

The same design twice: in the internal order with the die at the origin, and
with its nodes shuffled and the die moved (by a power of two, so that the
positions relative to the die are the same floats).  Every call gives the same
values node for node, with and without filler cells; a non-finite position
is refused and leaves the placement as it was.
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


def designs(ap, preset):
    """The design, its shuffled and moved copy, and the node order of the copy."""
    a = ap.synth.generate(preset, seed=3)
    rng = np.random.default_rng(5)
    n = len(a["node_w"])
    # movable cells keep their order among themselves, likewise the fixed ones:
    # the internal order (and with it every sum) is then the same
    order = np.argsort(np.concatenate([np.sort(rng.random(int((a["node_fixed"] == k).sum()))) for k in (0, 1)]),
                       kind="stable")  # copy's node i is a's node order[i]
    at = np.empty(n, np.int64)
    at[order] = np.arange(n)
    b = dict(a)
    for k in ("node_w", "node_h", "node_x", "node_y", "node_fixed"):
        b[k] = a[k][order]
    b["pin_node"] = at[a["pin_node"]].astype(np.int32)
    off = np.float32(1.0)
    b["node_x"], b["node_y"] = b["node_x"] + off, b["node_y"] + off
    b["die"] = a["die"] + off
    return a, b, order, off


def positions(nl, grid, seed):
    """Positions on multiples of 2^-8 (exact before and after the move)."""
    rng = np.random.default_rng(seed)
    x, y = nl["node_x"].copy(), nl["node_y"].copy()
    mov = nl["node_fixed"] == 0
    side = float(nl["die"][2]) - 40.0
    for v in (x, y):
        v[mov] = (rng.integers(0, int(side * 256), int(mov.sum())) / 256.0).astype(np.float32)
    return x, y


@pytest.mark.parametrize("fillers", [0, 1])
@pytest.mark.parametrize("preset", ["c0", "c1_small"])
def test_shuffled_and_moved_netlist(ap, preset, fillers):
    a, b, order, off = designs(ap, preset)
    if preset == "c0":
        a["die"] = np.array([0, 0, 64, 64], np.float32)
        b["die"] = a["die"] + off
    x, y = positions(a, 256, 9)
    xa, ya = np.round(a["node_x"] * 256) / 256, np.round(a["node_y"] * 256) / 256
    fixed = a["node_fixed"] == 1
    x[fixed], y[fixed] = xa[fixed], ya[fixed]
    a["node_x"], a["node_y"] = xa.astype(np.float32), ya.astype(np.float32)
    b["node_x"], b["node_y"] = a["node_x"][order] + off, a["node_y"][order] + off
    bx, by = x[order] + off, y[order] + off
    with ap.Placer(a, filler_cells=fillers) as p, ap.Placer(b, filler_cells=fillers) as q:
        m = p.params.bins_x
        for k, (u, v) in enumerate(zip(p.compute_all_partials(x, y, 3.0), q.compute_all_partials(bx, by, 3.0))):
            np.testing.assert_array_equal(u[order] if k < 2 else u, v)
        np.testing.assert_array_equal(p.compute_overlaps(x, y), q.compute_overlaps(bx, by))
        rng = np.random.default_rng(1)
        ex, ey = rng.standard_normal((2, m * m)).astype(np.float32)
        for u, v in zip(p.compute_node_forces(x, y, ex, ey), q.compute_node_forces(bx, by, ex, ey)):
            np.testing.assert_array_equal(u[order], v)
            assert not u[fixed].any()
        for u, v in zip(p.compute_node_forces(x, y, ex, ey, 3.0, 0.1), q.compute_node_forces(bx, by, ex, ey, 3.0, 0.1)):
            np.testing.assert_array_equal(u[order], v)
        p.initialize_placement(x, y)
        q.initialize_placement(bx, by)
        for u, v, w in zip(p.positions(), q.positions(), (x, y)):
            np.testing.assert_array_equal(u, w)
            np.testing.assert_array_equal(v, w[order] + off)
        p.perform_iteration(3)
        q.perform_iteration(3)
        for u, v in zip(p.positions(), q.positions()):
            np.testing.assert_array_equal(u[order] + off, v)
        assert p.stats()["hpwl"] == q.stats()["hpwl"]


def test_non_finite_positions_leave_the_placement(ap):
    nl = ap.synth.generate("c0", seed=1)
    with ap.Placer(nl) as p:
        p.initialize_placement(nl["node_x"], nl["node_y"])
        p.perform_iteration(2)
        before = p.positions(), p.stats()
        x = nl["node_x"].copy()
        x[5] = np.inf
        gx = np.zeros(64 * 64, np.float32)
        for call in (lambda: p.initialize_placement(x, nl["node_y"]),
                     lambda: p.compute_all_partials(x, nl["node_y"], 1.0),
                     lambda: p.compute_overlaps(nl["node_x"], x),
                     lambda: p.compute_node_forces(x, nl["node_y"], gx, gx)):
            with pytest.raises(ap.APError) as e:
                call()
            assert e.value.status == AP_ERR_NONFINITE
        after = p.positions(), p.stats()
        np.testing.assert_array_equal(before[0], after[0])
        assert before[1] == after[1]
        pad = np.flatnonzero(nl["node_fixed"] == 1)[0]
        x = nl["node_x"].copy()
        x[pad] = np.nan  # a fixed node's entry is ignored by the initial placement
        p.initialize_placement(x, nl["node_y"])

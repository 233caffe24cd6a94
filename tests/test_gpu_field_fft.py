"""The FP32 field solve by fast transforms, at every length it is built for.

Every power of two a handle takes (32 .. 4096; one, two or three radix-8
stages and a last one of 2, 4 or 8) and the lengths 2^k p of the
allocation-free call (p = 3, 5, 7), against the transforms in 64 bits, on a
rectangular grid.  Bound on the 2-norm, from the standard analysis of an FFT
in floating point (N. Higham, Accuracy and Stability of Numerical
Algorithms, 2nd ed., theorem 24.2): an FFT of length m errs by at most about
6.7 u log2(m), u = 2^-24; the reordering's twiddle before or after it adds a few u
(8 here); the solve runs four of them one after another:
4 u (6.7 log2(m) + 8).
"""
import ctypes as C
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


def bound(m):
    return 4.0 * 2.0 ** -24 * (6.7 * math.log2(m) + 8.0)


def exact(d, m, ratio):
    import torch

    k = torch.arange(m, dtype=torch.float64, device="cuda")
    t = torch.outer(k, k + 0.5) * (math.pi / m)
    c, s = torch.cos(t), torch.sin(t)
    w = k * (math.pi / m)
    wx, wy = w[:, None], w[None, :] * ratio
    a = c @ torch.from_numpy(d).cuda().double() @ c.T * (4.0 / m ** 2)
    a[0, :] *= 0.5
    a[:, 0] *= 0.5
    den = wx ** 2 + wy ** 2
    den[0, 0] = 1.0
    a[0, 0] = 0.0
    phi = a / den
    return (s.T @ (phi * wx) @ c).cpu().numpy(), (c.T @ (phi * wy) @ s).cpu().numpy()


def density(m, seed):
    rng = np.random.default_rng(seed)
    d = 0.1 * rng.standard_normal((m, m))
    d[m // 3: m // 2, m // 4: m // 2] += 2.5
    return (d - d.mean()).astype(np.float32)


def check(got, ref, m):
    for g, r in zip(got, ref):
        err = np.linalg.norm(g.reshape(m, m) - r) / np.linalg.norm(r)
        print(f"m {m}: {err:.2e} of the 2-norm, bound {bound(m):.2e}")
        assert err <= bound(m)


@pytest.mark.parametrize("m", [32, 64, 128, 256, 512, 1024, 2048, 4096])
def test_handle_solve(ap, m):
    nl = dict(ap.synth.generate("c0", seed=1))
    side = float(nl["die"][2])
    nl["die"] = np.array([0.0, 0.0, side, 1.5 * side], np.float32)
    bw, bh = np.float32(side) / np.float32(m), np.float32(1.5 * side) / np.float32(m)
    d = density(m, m)
    with ap.Placer(nl, bins=m) as pl:
        check(pl.compute_electric_fields(d, "fp32"), exact(d, m, float(bh / bw)), m)


@pytest.mark.parametrize("offset", [0, 1])  # outputs on an 8-byte boundary, and on a 4-byte one only
@pytest.mark.parametrize("m", [32, 64, 96, 128, 160, 192, 224, 256])
def test_device_buffer_solve(ap, m, offset):
    import torch

    from aieplace_gb300._lib import lib

    d = density(m, 7 * m)
    dd = torch.from_numpy(d).cuda()
    out = [torch.full((m * m + 2,), float("nan"), device="cuda") for _ in range(2)]
    ex, ey = (o[offset: offset + m * m] for o in out)
    st = lib().ap_field_solve_noalloc(C.c_void_p(dd.data_ptr()), C.c_void_p(ex.data_ptr()), C.c_void_p(ey.data_ptr()),
                                      m, C.c_float(0.75), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    torch.cuda.synchronize()
    check((ex.cpu().numpy(), ey.cpu().numpy()), exact(d, m, 0.75), m)
    for o in out:  # nothing outside the maps is written
        assert torch.isnan(o[:offset]).all() and torch.isnan(o[offset + m * m:]).all()


def test_batch_of_several_grids_matches_single_instances(ap):
    """Grids of 32 .. 2048 bins in one persistent launch (2048: only its
    larger block serves), bit for bit the instances alone."""
    nls = []
    for i, (cells, bins) in enumerate([(600, 32), (700, 64), (3000, 128), (5000, 256), (9000, 512), (2500, 1024),
                                       (2600, 2048)]):
        spec = dict(ap.synth.batch_specs(1, seed=i, lo=cells, hi=cells)[0], bins=bins)
        nls.append(ap.synth.generate(spec, seed=30 + i))
    for part in (nls[:6], nls):
        with ap.BatchPlacer(part) as b:
            b.initialize_placement(seed=50, sigma=1.0)
            b.step(5)
            got = [(b.positions(i), b.stats(i)["hpwl"]) for i in range(len(part))]
            info = b.info()
        assert info["form"] == "persistent" and info["field_tile"] in (32, 64)
        assert len(part) == 6 or info["field_tile"] == 64
        for i, nl in enumerate(part):
            with ap.Placer(nl, block_nodes=2048) as pl:
                pl.initialize_placement(seed=50 + i, sigma=1.0)
                pl.step_async(5)
                (x, y), hpwl = pl.positions(), pl.stats()["hpwl"]
            np.testing.assert_array_equal(got[i][0][0], x)
            np.testing.assert_array_equal(got[i][0][1], y)
            assert got[i][1] == hpwl

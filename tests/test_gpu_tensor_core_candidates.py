"""Every candidate of the tensor-core field solve, pinned with AP_TC_VARIANT at
create: without a pin the mixed-precision solver runs the FP32 fast transforms, so
a test that only asks for "bf16x3" does not reach the tcgen05 kernels.

  parity      max|dE| <= 1e-4 max|E| against the FP64 oracle, 128 to 1024 bins (the
              bound of every field test)
  scaling     E(2 d) = 2 E(d) within 1e-6 of max: doubling is exact in BF16 and FP32,
              so both solves make the same roundings
  repeatable  twelve more solves bit for bit (split-K partials summed in a fixed
              order)
  timeout     the load issuer told to issue nothing (ap_debug_inject): the bounded
              waits run out, the calls report AP_ERR_TIMEOUT, and without the
              injection the handle solves again bit for bit
  loop        20k cells on 128 bins to overflow < 0.10: the final HPWL within 0.5% and
              the overflow within 0.005 of the FP64 oracle loop's, as for the other
              solvers (test_gpu_parity.py)

The persistent candidates' (3, 4) agreement with the four launches, their timeout
and their loop against the FP32 one are in test_gpu_field_persistent.py.
"""
import numpy as np
import pytest

from test_gpu_field_persistent import AP_ERR_TIMEOUT, ap, density_like, pinned  # noqa: F401
from test_gpu_parity import clustered_start

pytestmark = pytest.mark.gpu

CANDIDATES = (0, 1, 2, 3, 4)
LAUNCHES = (0, 1, 2)  # four launches a solve


@pytest.mark.parametrize("m", [128, 256, 512, 1024])
@pytest.mark.parametrize("variant", CANDIDATES)
def test_candidate_field_against_oracle(ap, oracle_lib, monkeypatch, variant, m):
    d = density_like(m, np.random.default_rng(700 + m))
    nl = ap.synth.generate("c0", seed=1)
    with pinned(ap, monkeypatch, variant, nl, bins=m) as pl:
        ex, ey = pl.compute_electric_fields(d, "bf16x3")
        for _ in range(12):
            ex2, ey2 = pl.compute_electric_fields(d, "bf16x3")
            np.testing.assert_array_equal(ex2, ex)
            np.testing.assert_array_equal(ey2, ey)
        dx, dy = pl.compute_electric_fields(2.0 * d, "bf16x3")
        fx, _ = pl.compute_electric_fields(d, "fp32")
    assert not np.array_equal(ex, fx)  # not the transforms under another name
    solve = oracle_lib.field_solve_fft if m >= 512 else oracle_lib.field_solve
    rex, rey = solve(d.astype(np.float64), m)
    for got, twice, ref in ((ex, dx, rex), (ey, dy, rey)):
        ref = ref.reshape(got.shape)
        assert np.abs(got - ref).max() <= 1e-4 * np.abs(ref).max()
        assert np.abs(twice - 2 * got).max() <= 1e-6 * np.abs(got).max()


@pytest.mark.parametrize("m", [128, 512])
@pytest.mark.parametrize("variant", LAUNCHES)
def test_candidate_wait_runs_out_and_reports_timeout(ap, monkeypatch, variant, m):
    from aieplace_gb300 import APError
    from aieplace_gb300._lib import check, lib

    def inject(pl, kind, wait_ns=0):
        check("ap_debug_inject", lib().ap_debug_inject(pl._h, kind, wait_ns))

    d = density_like(m, np.random.default_rng(11))
    nl = ap.synth.generate("c1_small", seed=1)
    with pinned(ap, monkeypatch, variant, nl, bins=m, field_solver="bf16x3") as pl:
        pl.initialize_placement(seed=2, sigma=1.0)
        ex0, ey0 = pl.compute_electric_fields(d, "bf16x3")
        for call in (lambda: pl.compute_electric_fields(d, "bf16x3"), lambda: pl.perform_iteration(1)):
            inject(pl, 1, 10_000_000)  # AP_FAULT_TC_STALL, 10 ms per wait
            with pytest.raises(APError) as e:
                call()
            assert e.value.status == AP_ERR_TIMEOUT
            inject(pl, 0)
        ex1, ey1 = pl.compute_electric_fields(d, "bf16x3")
    np.testing.assert_array_equal(ex0, ex1)
    np.testing.assert_array_equal(ey0, ey1)


@pytest.fixture(scope="module")
def oracle_loop(ap, oracle_lib):
    nl = ap.synth.generate("c1_small", seed=1)
    x, y = clustered_start(nl, 1)
    ref = oracle_lib.Placer(nl, 128, 0.7)
    ref.init(x, y)
    while ref.stats()["overflow"] >= 0.10 and ref.stats()["iteration"] < 4000:
        ref.step(1)
    return nl, x, y, ref.stats()


@pytest.mark.parametrize("variant", CANDIDATES)
def test_candidate_loop_matches_oracle(ap, oracle_loop, monkeypatch, variant):
    nl, x, y, ref = oracle_loop
    with pinned(ap, monkeypatch, variant, nl, bins=128, target_density=0.7, check_interval=1,
                field_solver="bf16x3") as pl:
        pl.initialize_placement(x, y)
        pl.run()
        s = pl.stats()
    assert s["overflow"] < 0.10 and ref["overflow"] < 0.10, (s, ref)
    assert abs(s["hpwl"] - ref["hpwl"]) <= 0.005 * ref["hpwl"], (s, ref)
    assert abs(s["overflow"] - ref["overflow"]) <= 0.005, (s, ref)

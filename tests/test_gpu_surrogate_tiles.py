"""The surrogate's training pass by tiles ((K0, 1, 1, 1) nets) at the edges of
its shapes: three, six and eighteen input channels (factors 1, 2, 4), widths that are
not a multiple of a thread's four channels, maps of two and three tiles a
side, with and without a margin, against the FP64 oracle; tolerances as in
test_gpu_surrogate.py (FP32 sums of a map's pixels per weight): loss 1e-5
relative, gradient 1e-3 of its largest entry, cosine 0.99999.
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


@pytest.mark.parametrize("factor,k0,width,batch,res,margin", [
    (1, 1, 1, 1, 32, 0), (1, 3, 17, 3, 48, 5), (2, 1, 30, 1, 32, 1), (4, 3, 32, 2, 32, 0), (4, 1, 7, 1, 48, 15)])
def test_tile_gradient_matches_oracle(ap, oracle_lib, factor, k0, width, batch, res, margin):
    rng = np.random.default_rng(100 * factor + width)
    kernels = (k0, 1, 1, 1)
    with ap.Surrogate(factor=factor, kernels=kernels, width=width) as s:
        p = (0.15 * rng.standard_normal(s.num_params)).astype(np.float32)
        s.set_params(p)
        x = rng.standard_normal((batch, s.cin, res, res)).astype(np.float32)
        t = rng.standard_normal((batch, s.cout, res, res)).astype(np.float32)
        loss, g = s.gradient(x, t, margin)
        loss2, g2 = s.gradient(x, t, margin)
        np.testing.assert_array_equal(g, g2)
        assert loss == loss2
        y = s.forward(x)
        assert s.gradient(x, y, margin)[0] == 0.0  # training and inference forward: the same bits
        lr, gr = oracle_lib.surr_loss_grad(x, t, p.astype(np.float64), width, kernels, margin)
    assert abs(loss - lr) <= 1e-5 * lr
    assert np.abs(g - gr).max() <= 1e-3 * np.abs(gr).max()
    assert float(g @ gr) / (np.linalg.norm(g) * np.linalg.norm(gr)) >= 0.99999

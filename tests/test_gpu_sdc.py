"""nfft_sdc_weights (sdc.cu) against the oracle's sdc and against the same
iterations through the plan's real convolutions: both precisions, 1-D to 3-D,
tiled, plain and compensated plans, work arrays passed or not, zero iterations,
and non-positive sums.  Tolerance: 1e-5 (FP32), 1e-10 (FP64), as for the other
iterated convolutions of the suite (20 iterations of sums good to 1e-11)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402
from nfftgb300 import tools  # noqa: E402
from oracle import oracle  # noqa: E402


def by_convolutions(p, iters):
    w = torch.ones(p.J, dtype=p.dtype, device="cuda")
    t = torch.empty_like(w)
    g = nf.empty_image(p.Ntilde, p.dtype)
    for i in range(iters):
        p.convolve_transpose_(w, g)
        if i == 0:
            s = g.max()
        g.div_(s)
        p.convolve_(g, t)
        t.div_(s)
        w.div_(t)
    return w, t, g


@pytest.mark.parametrize("N,M", [((700,), 900), ((24, 31), 1500), ((12, 10, 9), 1300)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kw", [{}, {"blocking": False}, {"compensated": True}])
def test_sdc_weights(N, M, dtype, kw):
    rng = np.random.default_rng(M)
    k = (rng.random((len(N), M)) - 0.5).astype(dtype)
    p = nf.plan_nfft(k, N, m=4, sigma=2.0, precompute=nf.TENSOR, **kw)
    tol = 1e-5 if dtype == np.float32 else 1e-10
    w_ref, t_ref, g_ref = by_convolutions(p, 7)
    w = torch.ones(M, dtype=p.dtype, device="cuda")
    t = torch.empty_like(w)
    g = nf.empty_image(p.Ntilde, p.dtype)
    scaled = tools.sdc(p, iters=7, weights=w, weights_tmp=t, workg=g)
    assert scaled is w
    op = oracle.OraclePlan(k.astype(np.float64), N, m=4, sigma=2.0, precompute=oracle.TENSOR)
    assert oracle.rel_l2(w.cpu().numpy(), oracle.sdc(op, iters=7)) < tol
    ratio = w.double() / w_ref.double()  # up to the final scaling
    assert float((ratio / ratio.mean() - 1).abs().max()) < 20 * tol
    assert oracle.rel_l2(t.cpu().numpy(), t_ref.cpu().numpy()) < tol
    assert oracle.rel_l2(g.cpu().numpy().ravel(order="F"), g_ref.cpu().numpy().ravel(order="F")) < tol
    assert oracle.rel_l2(tools.sdc(p, iters=7).cpu().numpy(), w.cpu().numpy()) < tol


def test_sdc_edges():
    k = (np.random.default_rng(2).random((2, 60)) - 0.5).astype(np.float32)
    p = nf.plan_nfft(k, (16, 16), m=4, sigma=2.0, precompute=nf.TENSOR)
    w = torch.ones(60, device="cuda")
    w[7] = -1e6  # its own sum is negative
    with pytest.raises(ValueError, match="non-positive weights"):
        tools.sdc(p, iters=3, weights=w)
    assert tools.sdc(p, iters=0).shape == (60,)
    with pytest.raises(nf.DimensionMismatch):
        tools.sdc(p, weights=torch.ones(61, device="cuda"))
    with pytest.raises(nf.ArgumentError):
        tools.sdc(p, weights=torch.ones(60, dtype=torch.float64, device="cuda"))

"""nfft_sdc_weights when some sum is not positive: weights, weights_tmp and workg
hold what the same iterations through the plan's convolutions hold where they stop
(before the division).

A weight of -1.2 (-1.0) beside a node 0.3 grid cells away makes its sum negative in
the fourth (sixth) iteration, -1e6 in the first; the number of iterations puts
the stop in the last, the last but one, and an earlier one.  Tolerances as in
the other sdc tests, times 10 for sums that cancel; weights that were never
divided stay equal to the bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402
from nfftgb300 import tools  # noqa: E402
from oracle import oracle  # noqa: E402


def until_stop(p, w, iters):
    t = torch.empty_like(w)
    g = nf.empty_image(p.Ntilde, p.dtype)
    for i in range(iters):
        p.convolve_transpose_(w, g)
        if i == 0:
            s = g.max()
        g.div_(s)
        p.convolve_(g, t)
        t.div_(s)
        if bool((t <= 0).any()):
            return i, t, g
        w.div_(t)
    return None, t, g


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("value,iters,stop", [(-1.2, 9, 3), (-1.2, 5, 3), (-1.2, 4, 3), (-1.0, 20, 5), (-1e6, 3, 0),
                                              (-1e6, 1, 0)])
@pytest.mark.parametrize("kw", [{}, {"blocking": False}])
def test_state_where_the_iterations_stop(dtype, value, iters, stop, kw):
    k = (np.random.default_rng(2).random((2, 60)) - 0.5).astype(np.float32).astype(dtype)
    p = nf.plan_nfft(k, (16, 16), m=4, sigma=2.0, precompute=nf.TENSOR, **kw)
    start = torch.ones(60, dtype=p.dtype, device="cuda")
    start[31] = value
    w_ref = start.clone()
    i, t_ref, g_ref = until_stop(p, w_ref, iters)
    assert i == stop
    w, t = start.clone(), torch.zeros_like(start)
    g = nf.empty_image(p.Ntilde, p.dtype)
    with pytest.raises(ValueError, match="non-positive weights"):
        tools.sdc(p, iters=iters, weights=w, weights_tmp=t, workg=g)
    tol = 1e-4 if dtype == np.float32 else 1e-9
    if stop == 0:
        assert torch.equal(w, start)
    assert oracle.rel_l2(w.cpu().numpy(), w_ref.cpu().numpy()) < tol
    assert oracle.rel_l2(t.cpu().numpy(), t_ref.cpu().numpy()) < tol
    assert oracle.rel_l2(g.cpu().numpy().ravel(), g_ref.cpu().numpy().ravel()) < tol
    w2 = start.clone()  # without work arrays
    with pytest.raises(ValueError):
        tools.sdc(p, iters=iters, weights=w2)
    assert oracle.rel_l2(w2.cpu().numpy(), w_ref.cpu().numpy()) < tol


def test_number_of_iterations_as_in_a_range():
    k = (np.random.default_rng(2).random((2, 60)) - 0.5).astype(np.float32)
    p = nf.plan_nfft(k, (16, 16), m=4, sigma=2.0, precompute=nf.TENSOR)
    none = tools.sdc(p, iters=0)
    assert oracle.rel_l2(tools.sdc(p, iters=-3).cpu().numpy(), none.cpu().numpy()) < 1e-5
    assert oracle.rel_l2(tools.sdc(p, iters=np.int64(0)).cpu().numpy(), none.cpu().numpy()) < 1e-5
    with pytest.raises(TypeError):
        tools.sdc(p, iters=2.5)

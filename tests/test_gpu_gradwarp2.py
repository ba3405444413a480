"""The tiled 2-D node gradient (gradwarp2.cuh): every m, window modes, both
precisions, ragged tiles that wrap, a hot tile, and a sparse set (warp-per-node
kernel).

Against the exact gradient (FP64 NDFT), POLYNOMIAL and FULL: the NFFT's
derivative carries the window's truncation error times Ntilde, at most 50 x the
forward error bound of test/accuracy.jl for m (10^-(1.5 m - 1) covers
Kaiser-Bessel at sigma = 2), floored at the FP32 bar 2e-5.  Against the
warp-per-node kernel (blocking = False), all modes: the same window values and
derivatives, other orders of summation and another FFT (centred grid), 5e-5 /
1e-11.  (The derivative of the LUT's linear interpolant is a difference quotient
over LUTSize/m steps per unit, so in FP32 it has no better value to compare with
than itself.)"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402
from oracle import oracle  # noqa: E402


def exact_gradient(k, f, w):
    n = [np.arange(s) - s // 2 for s in f.shape]
    e = [np.exp(-2j * np.pi * np.outer(k[d], n[d])) for d in range(2)]
    out = np.zeros_like(k)
    for d in range(2):
        ed = list(e)
        ed[d] = ed[d] * (-2j * np.pi * n[d])[None]
        out[d] = np.real(np.conj(w) * np.einsum("ja,ab,jb->j", ed[0], f, ed[1]))
    return out


def problem(N, M, m, dtype):
    rng = np.random.default_rng(m + M)
    k = rng.random((2, M)) - 0.5
    k[:, :3] = [[-0.5, 0.4999, 0.0], [0.25, -0.5, 0.4999]]
    if M > 1000:
        k[:, 50:50 + 333] = 0.11 + 0.001 * rng.random((2, 333))
    f = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    w = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    return k.astype(dtype), f, w


def gradient(k, f, w, **kw):
    p = nf.plan_nfft(k, f.shape, sigma=2.0, **kw)
    buf = torch.empty((k.shape[1], 2), dtype=p.dtype, device="cuda")
    p.grad_nodes_(buf.t(), nf.as_colmajor(f, f.shape, p.cdtype), torch.as_tensor(w).to(p.cdtype).cuda())
    return buf.t().cpu().numpy()


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("pre", [nf.POLYNOMIAL, nf.FULL])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("N,M", [((40, 27), 3000), ((60, 50), 23)])
def test_gradient(m, pre, dtype, N, M):
    k, f, w = problem(N, M, m, dtype)
    got = gradient(k, f, w, m=m, precompute=pre)
    ref = exact_gradient(k.astype(np.float64), f, w)
    tol = 50 * 10.0 ** -(1.5 * m - 1)
    tol = max(tol, 2e-5 if dtype == np.float32 else 1e-9)
    assert oracle.rel_l2(got, ref) < tol


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("pre", [nf.TENSOR, nf.FULL, nf.LINEAR])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_gradient_equals_the_general_path(m, pre, dtype):
    k, f, w = problem((40, 27), 3000, m, dtype)
    a = gradient(k, f, w, m=m, precompute=pre)
    b = gradient(k, f, w, m=m, precompute=pre, blocking=False)
    assert oracle.rel_l2(a, b) < (5e-5 if dtype == np.float32 else 1e-11)

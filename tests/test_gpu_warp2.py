"""The one-warp-per-task 2-D spreader and gather (warp2.cuh) against the oracle.

Sizes where they can go wrong: every m (2m x 2m taps: full and partial last
steps), both precisions, table and polynomial windows; ragged tiles that wrap;
grids smaller than the window; a hot tile split into chunks with a remainder;
node sets too sparse for the tiled gather.  Tolerances: the suite's parity bars
(1e-11 for FP64, 1e-5 for FP32); FP64 polynomial windows with m >= 6 differ by
the conditioning of two least-squares fits of degree 2m, eps x ~1e6 = 1e-10."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402
from oracle import oracle  # noqa: E402

PROBLEMS = {
    "ragged": ((70, 45), 6000, None),
    "tiny grid": ((3, 5), 700, None),
    "sparse": ((200, 180), 37, None),
    "wide tiles": ((70, 45), 4500, (40, 24)),
}


def nodes(N, M, dtype):
    rng = np.random.default_rng(M)
    k = rng.random((2, M)) - 0.5
    k[:, :4] = [[-0.5, 0.4999, 0.0, 0.25], [0.4999, -0.5, -0.001, -0.5]]
    if M > 1000:  # a hot tile: several chunks and a remainder of one node
        k[:, 100:100 + 577] = 0.11 + 0.001 * rng.random((2, 577))
    return k.astype(dtype), rng


@pytest.mark.parametrize("problem", PROBLEMS)
@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("pre", [oracle.FULL, oracle.POLYNOMIAL])
def test_warp2_matches_oracle(problem, m, dtype, pre):
    N, M, bs = PROBLEMS[problem]
    k, rng = nodes(N, M, dtype)
    f = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    v = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    p = nf.plan_nfft(k, N, m=m, sigma=2.0, precompute=pre, **({"blockSize": bs} if bs else {}))
    op = oracle.OraclePlan(k.astype(np.float64), N, m=m, sigma=2.0, precompute=pre)
    tol = 1e-5 if dtype == np.float32 else (1e-10 if pre == oracle.POLYNOMIAL and m >= 6 else 1e-11)
    f, v = f.astype(np.complex64), v.astype(np.complex64)  # the same inputs in both precisions
    y = (p * nf.as_colmajor(f, N, p.cdtype)).cpu().numpy()
    x = (nf.adjoint(p) * torch.as_tensor(v).to(p.cdtype)).cpu().numpy()
    assert oracle.rel_l2(y, op.forward(f.astype(np.complex128))) < tol
    assert oracle.rel_l2(x.ravel(order="F"), op.adjoint(v.astype(np.complex128)).ravel(order="F")) < tol


@pytest.mark.parametrize("m", [3, 4, 5])
def test_warp2_columns(m):
    """Multi-column launches (directional plans): each column equals its single 2-D plan."""
    N, M, C = (40, 36), 3000, 5
    k, rng = nodes(N, M, np.float32)
    f = nf.as_colmajor((rng.standard_normal(N + (C,)) + 1j * rng.standard_normal(N + (C,))).astype(np.complex64),
                       N + (C,), torch.complex64)
    v = nf.as_colmajor((rng.standard_normal((M, C)) + 1j * rng.standard_normal((M, C))).astype(np.complex64),
                       (M, C), torch.complex64)
    p = nf.plan_nfft(k, N + (C,), dims=(1, 2), m=m, sigma=2.0)
    one = nf.plan_nfft(k, N, m=m, sigma=2.0, precompute=nf.LINEAR)
    y, x = p * f, nf.adjoint(p) * v
    for c in range(C):
        assert oracle.rel_l2(y[:, c].cpu().numpy(), (one * f[:, :, c]).cpu().numpy()) < 1e-5
        assert oracle.rel_l2(x[:, :, c].cpu().numpy(), (nf.adjoint(one) * v[:, c].contiguous()).cpu().numpy()) < 1e-5


@pytest.mark.parametrize("N,C", [((32, 32), 3), ((64, 128), 7), ((256, 64), 65), ((512, 32), 2)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_fused_columns(monkeypatch, N, C, dtype):
    """Directional plans with power-of-two grids run the pruned line FFTs over
    all columns; each column equals the cuFFT path's."""
    k, rng = nodes(N, 900, dtype)
    cd = torch.complex64 if dtype == np.float32 else torch.complex128
    f = nf.as_colmajor(rng.standard_normal(N + (C,)) + 1j * rng.standard_normal(N + (C,)), N + (C,), cd)
    v = nf.as_colmajor(rng.standard_normal((900, C)) + 1j * rng.standard_normal((900, C)), (900, C), cd)
    p = nf.plan_nfft(k, N + (C,), dims=(1, 2), m=4, sigma=2.0)
    y, x = (p * f).cpu().numpy(), (nf.adjoint(p) * v).cpu().numpy()
    monkeypatch.setenv("NFFT_GB300_FFT", "cufft")
    q = nf.plan_nfft(k, N + (C,), dims=(1, 2), m=4, sigma=2.0)
    ref_y, ref_x = (q * f).cpu().numpy(), (nf.adjoint(q) * v).cpu().numpy()
    tol = 1e-5 if dtype == np.float32 else 1e-11
    for c in range(C):
        assert oracle.rel_l2(y[:, c], ref_y[:, c]) < tol
        assert oracle.rel_l2(x[:, :, c], ref_x[:, :, c]) < tol

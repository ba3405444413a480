"""The 1-D gather and sorting spreader (line1.cuh) against the oracle.

Every m, both precisions, table and polynomial windows, plain and compensated
sums; node counts around a warp, a sort batch (512) and a task (2048); a hot
cell; a grid smaller than the window; a last tile that is not whole; tiles
larger than the sorting spreader takes; sparse sets (direct gather).
Tolerances: the suite's parity bars, 1e-11 (FP64; 1e-10 for polynomial windows
with m >= 6, the conditioning of two degree-2m fits) and 1e-5 (FP32)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402
from oracle import oracle  # noqa: E402


def check(N, M, m, dtype, pre, comp, bs=None, hot=0, seed=5):
    rng = np.random.default_rng(seed)
    k = rng.random((1, M)) - 0.5
    k[0, :min(3, M)] = [-0.5, 0.4999, 0.0][:min(3, M)]
    if hot:
        k[0, 3:3 + hot] = 0.1 + 1e-3 * rng.random(hot) / N
    k = k.astype(dtype)
    f = (rng.standard_normal(N) + 1j * rng.standard_normal(N)).astype(np.complex64)
    v = (rng.standard_normal(M) + 1j * rng.standard_normal(M)).astype(np.complex64)
    p = nf.plan_nfft(k, (N,), m=m, sigma=2.0, precompute=pre, compensated=comp,
                     **({"blockSize": (bs,)} if bs else {}))
    op = oracle.OraclePlan(k.astype(np.float64), (N,), m=m, sigma=2.0, precompute=pre)
    tol = 1e-5 if dtype == np.float32 else (1e-10 if pre == oracle.POLYNOMIAL and m >= 6 else 1e-11)
    y = (p * nf.as_colmajor(f, (N,), p.cdtype)).cpu().numpy()
    x = (nf.adjoint(p) * torch.as_tensor(v).to(p.cdtype)).cpu().numpy()
    assert oracle.rel_l2(y, op.forward(f.astype(np.complex128))) < tol
    assert oracle.rel_l2(x, op.adjoint(v.astype(np.complex128))) < tol


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("pre", [oracle.FULL, oracle.TENSOR, oracle.POLYNOMIAL])
@pytest.mark.parametrize("comp", [False, True])
def test_line_matches_oracle(m, dtype, pre, comp):
    check(1500, 9000, m, dtype, pre, comp, hot=700)


@pytest.mark.parametrize("M", [1, 31, 33, 511, 513, 2047, 2050])
@pytest.mark.parametrize("comp", [False, True])
def test_line_node_counts(M, comp):
    check(64, M, 4, np.float32, oracle.POLYNOMIAL, comp, bs=128)   # one tile: M nodes in one task


@pytest.mark.parametrize("bs", [8, 37, 1024, 3000])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_line_tiles(bs, dtype):
    for comp in (False, True):
        check(1999, 6000, 5, dtype, oracle.TENSOR, comp, bs=bs)
    check(3, 50, 5, dtype, oracle.POLYNOMIAL, True)                  # the window exceeds the grid
    check(50000, 40, 4, dtype, oracle.POLYNOMIAL, False, bs=bs)      # sparse

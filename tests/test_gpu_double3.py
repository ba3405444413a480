"""The 3-D FP64 gather and spreader (double3.cuh) against the oracle.

Every m, table and polynomial windows, the default and other tile shapes, a
grid that is no whole number of tiles and wraps, a grid smaller than the window,
a hot tile of several batches with a remainder, and sets too sparse for the
tiled gather.  Tolerance: the suite's FP64 bar, 1e-11 (1e-10 for polynomial
windows with m >= 6: the conditioning of two least-squares fits of degree 2m)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402
from oracle import oracle  # noqa: E402


def check(N, M, m, pre, bs=None):
    rng = np.random.default_rng(M + m)
    k = rng.random((3, M)) - 0.5
    k[:, :4] = [[-0.5, 0.4999, 0.0, 0.25]] * 3
    if M > 2000:
        k[:, 50:50 + 181] = 0.2 + 0.002 * rng.random((3, 181))
    f = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    v = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    p = nf.plan_nfft(k, N, m=m, sigma=2.0, precompute=pre, **({"blockSize": bs} if bs else {}))
    op = oracle.OraclePlan(k, N, m=m, sigma=2.0, precompute=pre)
    tol = 1e-10 if pre == oracle.POLYNOMIAL and m >= 6 else 1e-11
    y = (p * nf.as_colmajor(f, N, torch.complex128)).cpu().numpy()
    assert oracle.rel_l2(y, op.forward(f)) < tol
    try:
        x = (nf.adjoint(p) * torch.as_tensor(v)).cpu().numpy()
    except NotImplementedError as e:  # tiles of the widest windows exceed shared memory and are refused
        assert m >= 7 and "does not fit in shared memory" in str(e)
        return
    assert oracle.rel_l2(x.ravel(order="F"), op.adjoint(v).ravel(order="F")) < tol


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("pre", [oracle.FULL, oracle.POLYNOMIAL])
@pytest.mark.parametrize("bs", [None, (16, 8, 4), (8, 8, 8), (5, 7, 3)])
def test_double3_matches_oracle(m, pre, bs):
    check((23, 17, 20), 4000, m, pre, bs)


@pytest.mark.parametrize("m", [2, 5, 8])
def test_double3_sparse_and_tiny(m):
    check((30, 28, 26), 45, m, oracle.POLYNOMIAL)
    check((3, 4, 5), 300, m, oracle.FULL)

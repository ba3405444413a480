"""Shared-memory limits of the tiled kernels: a kernel's limit belongs to the
function, not to the plan or batch that asked for it.

A batch with large tiles must still run after a batch with small tiles of the
same kernel was created (its kernels are launched at its first call, not at its
creation), for every kernel of the batch.  Tolerances: those of the batch tests,
each member against its own transforms."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402
from oracle import oracle  # noqa: E402


def member(N, M, dtype, bs, pre, seed):
    rng = np.random.default_rng(seed)
    k = (rng.random((len(N), M)) - 0.5).astype(dtype)
    p = nf.plan_nfft(k, N, m=4, sigma=2.0, precompute=pre, blockSize=bs)
    f = nf.as_colmajor(rng.standard_normal(N) + 1j * rng.standard_normal(N), N, p.cdtype)
    v = torch.as_tensor(rng.standard_normal(M) + 1j * rng.standard_normal(M)).to(device="cuda", dtype=p.cdtype)
    return p, f, v


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("pre", [nf.TENSOR, nf.POLYNOMIAL])
@pytest.mark.parametrize("N,large,small", [((64, 64), (96, 64), (8, 8)), ((24, 24, 24), (16, 16, 8), (8, 8, 4))])
def test_small_batch_does_not_lower_the_limit_of_a_large_one(dtype, pre, N, large, small):
    p, f, v = member(N, 6000, dtype, large, pre, 1)
    a = nf.NFFTBatch([p])
    q, g, w = member(N, 6000, dtype, small, pre, 2)
    b = nf.NFFTBatch([q])
    tol = 1e-12 if dtype == np.float64 else 1e-6
    for batch, plan, fi, vi in ((a, p, f, v), (b, q, g, w), (a, p, f, v)):
        y, x = batch.forward([fi])[0], batch.adjoint([vi])[0]
        assert oracle.rel_l2(y.cpu().numpy(), (plan * fi).cpu().numpy()) <= tol
        assert oracle.rel_l2(x.cpu().numpy(), (nf.adjoint(plan) * vi).cpu().numpy()) <= tol

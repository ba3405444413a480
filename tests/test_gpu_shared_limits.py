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


# Explicit FP64 tiles in the gap between the largest that the one-warp spreader (staging
# of 7,680 bytes at m = 2 to 26,112 at m = 8, table windows) and the two-warp one (5,888 to
# 21,248) can hold in 227 KB: m, block size, padded tile bytes = 16 (b0 + 2m - 1)(b1 + 2m - 1)
GAP = [(2, (71, 187)), (3, (70, 180)), (4, (61, 195)), (5, (60, 188)), (8, (47, 195))]


def gap_bytes(m, bs):
    return 16 * (bs[0] + 2 * m - 1) * (bs[1] + 2 * m - 1)


@pytest.mark.parametrize("m,bs", GAP)
def test_tiles_between_the_two_stagings(m, bs):
    """Single plans, stacks and batches with such tiles run, as with the larger spreader's limit before."""
    one = {2: 7680, 3: 10752, 4: 13824, 5: 16896, 8: 26112}[m]
    two = 32 * (8 + 16 * (2 * m + 1) + 8 * (6 * m))
    assert 227 * 1024 - one < gap_bytes(m, bs) <= 227 * 1024 - two - 32
    N, M, C = (120, 130), 9000, 3
    rng = np.random.default_rng(m)
    k = rng.random((2, M)) - 0.5
    f = nf.as_colmajor(rng.standard_normal(N + (C,)) + 1j * rng.standard_normal(N + (C,)), N + (C,), torch.complex128)
    v = nf.as_colmajor(rng.standard_normal((M, C)) + 1j * rng.standard_normal((M, C)), (M, C), torch.complex128)
    op = oracle.OraclePlan(k, N, m=m, sigma=2.0, precompute=oracle.FULL)
    tol = 1e-11
    fh, vh = f.cpu().numpy(), v.cpu().numpy()
    p = nf.plan_nfft(k, N, m=m, sigma=2.0, precompute=nf.FULL, blockSize=bs)
    y, x = (p * f[:, :, 0]).cpu().numpy(), (nf.adjoint(p) * v[:, 0]).cpu().numpy()
    ref_y, ref_x = op.forward(fh[:, :, 0]), op.adjoint(vh[:, 0])
    assert oracle.rel_l2(y, ref_y) < tol and oracle.rel_l2(x.ravel(order="F"), ref_x.ravel(order="F")) < tol
    batch = nf.NFFTBatch([p, nf.plan_nfft(k[:, :700], N, m=m, sigma=2.0, precompute=nf.FULL)])
    ys = batch.forward([nf.as_colmajor(f[:, :, 0], N, torch.complex128)] * 2)
    xs = batch.adjoint([v[:, 0].contiguous(), v[:700, 0].contiguous()])
    assert oracle.rel_l2(ys[0].cpu().numpy(), ref_y) < tol
    assert oracle.rel_l2(ys[1].cpu().numpy(), ref_y[:700]) < tol
    assert oracle.rel_l2(xs[0].cpu().numpy().ravel(order="F"), ref_x.ravel(order="F")) < tol
    # stacks evaluate their window by linear interpolation: against single plans that do so too
    q = nf.plan_nfft(k, N + (C,), dims=(1, 2), m=m, sigma=2.0, blockSize=bs)
    s = nf.plan_nfft(k, N, m=m, sigma=2.0, precompute=nf.LINEAR)
    ys, xs = (q * f).cpu().numpy(), (nf.adjoint(q) * v).cpu().numpy()
    for c in range(C):
        assert oracle.rel_l2(ys[:, c], (s * nf.as_colmajor(f[:, :, c], N, torch.complex128)).cpu().numpy()) < tol
        ref = (nf.adjoint(s) * v[:, c].contiguous()).cpu().numpy()
        assert oracle.rel_l2(xs[:, :, c].ravel(), ref.ravel()) < tol

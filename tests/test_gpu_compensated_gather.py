"""Gathers and node gradients of compensated plans, whose tasks are long: with tasks
of uneven length that do not fill the GPU they run a warp per node (as plans without
compensation do for sparse sets), with even ones or many the tiled kernels.  The
kernel is asserted, the values compared with the oracle at its bars, or, for many
nodes, with the FP64 plan (FP32 bar 1e-5)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402
from kernel_route import launched  # noqa: E402
from oracle import oracle  # noqa: E402

KERNELS = ("interp_kernel", "gather_warp2_kernel", "gather_plane3_kernel", "gather_double3_kernel", "interp_tile3_kernel",
           "grad_nodes_kernel", "grad_warp2_kernel")


def problem(N, M, dtype, seed):
    rng = np.random.default_rng(seed)
    D = len(N)
    k = rng.random((D, M)) - 0.5
    k[:, : M // 2] *= 0.15          # hot tiles: several tasks of 1024 nodes
    k = k.astype(dtype)
    f = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    v = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    return k, f.astype(np.complex64), v.astype(np.complex64)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("N,M,m", [((48, 40), 40000, 4), ((48, 40), 40000, 5), ((32, 28, 30), 66000, 3),
                                   ((32, 28, 30), 66000, 5)])
def test_long_tasks(dtype, N, M, m):
    k, f, v = problem(N, M, dtype, m)
    p = nf.plan_nfft(k, N, m=m, sigma=2.0, compensated=True)
    fd, y = nf.as_colmajor(f, N, p.cdtype), torch.empty(M, dtype=p.cdtype, device="cuda")
    nf.mul_(y, p, fd)
    assert launched(lambda: nf.mul_(y, p, fd), *KERNELS) == {"interp_kernel"}
    op = oracle.OraclePlan(k.astype(np.float64), N, m=m, sigma=2.0, precompute=oracle.POLYNOMIAL)
    tol = 1e-5 if dtype == np.float32 else 1e-11
    assert oracle.rel_l2(y.cpu().numpy(), op.forward(f.astype(np.complex128))) < tol
    if len(N) == 2:
        vd = torch.as_tensor(v).to(device="cuda", dtype=p.cdtype)
        dk, dq = (torch.empty((M, 2), dtype=p.dtype, device="cuda") for _ in range(2))
        p.grad_nodes_(dk.t(), fd, vd)
        assert launched(lambda: p.grad_nodes_(dk.t(), fd, vd), *KERNELS) == {"grad_nodes_kernel"}
        q = nf.plan_nfft(k, N, m=m, sigma=2.0, blocking=False)
        q.grad_nodes_(dq.t(), fd, vd)
        assert oracle.rel_l2(dk.cpu().numpy(), dq.cpu().numpy()) < (5e-5 if dtype == np.float32 else 1e-11)


@pytest.mark.parametrize("N,m,kernel", [((48, 40), 4, "gather_warp2_kernel"), ((18, 16, 14), 3, "gather_plane3_kernel"),
                                        ((18, 16, 14), 5, "gather_plane3_kernel")])
def test_many_nodes(N, m, kernel):
    M = 2**19 + 5
    k, f, v = problem(N, M, np.float32, m)
    p = nf.plan_nfft(k, N, m=m, sigma=2.0, compensated=True)
    q = nf.plan_nfft(k.astype(np.float64), N, m=m, sigma=2.0)
    fd, y = nf.as_colmajor(f, N, p.cdtype), torch.empty(M, dtype=p.cdtype, device="cuda")
    nf.mul_(y, p, fd)
    assert launched(lambda: nf.mul_(y, p, fd), *KERNELS) == {kernel}
    assert oracle.rel_l2(y.cpu().numpy(), (q * nf.as_colmajor(f, N, q.cdtype)).cpu().numpy()) < 1e-5


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("N,M,m,kernels", [((128, 128), 50000, 5, ("gather_warp2_kernel",) * 2),
                                           ((32, 32, 32), 66000, 5, ("gather_plane3_kernel", "gather_double3_kernel"))])
def test_even_tasks(dtype, N, M, m, kernels):
    _, f, _ = problem(N, M, dtype, m)
    k = (np.random.default_rng(3).random((len(N), M)) - 0.5).astype(dtype)
    p = nf.plan_nfft(k, N, m=m, sigma=2.0, compensated=True)
    fd, y = nf.as_colmajor(f, N, p.cdtype), torch.empty(M, dtype=p.cdtype, device="cuda")
    nf.mul_(y, p, fd)
    assert launched(lambda: nf.mul_(y, p, fd), *KERNELS) == {kernels[dtype is np.float64]}
    op = oracle.OraclePlan(k.astype(np.float64), N, m=m, sigma=2.0, precompute=oracle.POLYNOMIAL)
    tol = 1e-5 if dtype == np.float32 else 1e-11
    assert oracle.rel_l2(y.cpu().numpy(), op.forward(f.astype(np.complex128))) < tol

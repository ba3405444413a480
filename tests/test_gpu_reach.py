"""The tiled kernels with node counts past the rules that lead to them, over window
widths, table and polynomial windows, both precisions and tile shapes, each case
asserting that its kernel ran.

Against the oracle: 1e-5 (FP32), 1e-11 (FP64; 1e-10 for polynomial windows with
m >= 6, the conditioning of two least-squares fits of degree 2m).  1-D, FP32, m = 2
against the plan's plain path, 1e-5: a node within an FP32 rounding of a grid point may fall
into the cell beside the exact one, and the window of m = 2 ends with a step of 2e-3, so
a few nodes of the FP32 plan differ from the FP64 oracle by that, with any kernel."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402
from kernel_route import launched  # noqa: E402
from oracle import oracle  # noqa: E402

F32, F64 = np.float32, np.float64
TABLES = [oracle.TENSOR, oracle.FULL, oracle.POLYNOMIAL]


def nodes(D, M, dtype, hot, seed):
    rng = np.random.default_rng(seed)
    k = rng.random((D, M)) - 0.5
    edge = [-0.5, 0.4999, 0.0, -0.001, 0.25]
    k[:, :5] = [edge[d:] + edge[:d] for d in range(D)]
    if hot:  # a hot tile of several tasks, the last with a remainder
        k[:, 100:100 + hot] = 0.11 + 0.001 * rng.random((D, hot))
    return k.astype(dtype)


def check(direction, N, M, m, dtype, pre, kernels, hot=700, seed=1, **kw):
    """kernels: one of them must have run."""
    k = nodes(len(N), M, dtype, hot, seed)
    rng = np.random.default_rng(seed + 1)
    p = nf.plan_nfft(k, N, m=m, sigma=2.0, precompute=pre, **kw)
    op = oracle.OraclePlan(k.astype(np.float64), N, m=m, sigma=2.0, precompute=pre)
    tol = 1e-5 if dtype == F32 else (1e-10 if pre == oracle.POLYNOMIAL and m >= 6 else 1e-11)
    if direction == "forward":
        f = (rng.standard_normal(N) + 1j * rng.standard_normal(N)).astype(np.complex64)
        fd, got = nf.as_colmajor(f, N, p.cdtype), torch.empty(M, dtype=p.cdtype, device="cuda")
        call, ref = (lambda: nf.mul_(got, p, fd)), op.forward(f.astype(np.complex128))
    else:
        v = (rng.standard_normal(M) + 1j * rng.standard_normal(M)).astype(np.complex64)
        vd, got = torch.as_tensor(v).to(device="cuda", dtype=p.cdtype), nf.empty_image(N, p.cdtype)
        call, ref = (lambda: nf.mul_(got, nf.adjoint(p), vd)), op.adjoint(v.astype(np.complex128))
    if dtype == F32 and m == 2 and len(N) == 1:
        q = nf.plan_nfft(k, N, m=m, sigma=2.0, precompute=pre, blocking=False)
        ref = (q * fd if direction == "forward" else nf.adjoint(q) * vd).cpu().numpy()
    call()
    assert launched(call, *kernels)
    call()
    assert oracle.rel_l2(got.cpu().numpy().ravel(order="F"), ref.ravel(order="F")) < tol
    assert nf.load().nfft_sync(p._handle) == 0


# ---- 1-D
@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("pre", TABLES)
@pytest.mark.parametrize("comp", [False, True])
def test_sorting_spreader(m, dtype, pre, comp):
    """Whole and ragged tiles of 100 cells (33 batches of equal size and a hot cell)."""
    if not comp and (m <= 4 if dtype == F32 else m in (2, 8)):
        pytest.skip("spread by atomics")
    M = 2**20 + 77 if dtype == F64 and m >= 5 else 70001
    check("adjoint", (1499,), M, m, dtype, pre, ["spread_line_kernel"], compensated=comp, blockSize=(100,))


@pytest.mark.parametrize("chunk", [33, 511, 513, 1025, 2047])
@pytest.mark.parametrize("bs", [64, 101, 1024])
@pytest.mark.parametrize("dtype,comp", [(F32, True), (F32, False), (F64, True)])
def test_sorting_spreader_batches(monkeypatch, chunk, bs, dtype, comp):
    """Tasks around one and two batches of 512 nodes, tiles up to the largest."""
    monkeypatch.setenv("NFFT_GB300_TASK_CHUNK", str(chunk))
    m = 5 if dtype == F32 else 4
    check("adjoint", (999,), 66001, m, dtype, oracle.POLYNOMIAL, ["spread_line_kernel"], compensated=comp, blockSize=(bs,))


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("pre", TABLES)
def test_line_gather_from_tiles(m, dtype, pre):
    table = pre == oracle.FULL or (pre == oracle.TENSOR and dtype == F64)  # (FP32 TENSOR: Horner)
    kernel = "gather_line_kernelILi%dE%sLb%dELb1E" % (2 * m, "f" if dtype == F32 else "d", table)
    check("forward", (1499,), 140001 if dtype == F64 else 20001, m, dtype, pre, [kernel], blockSize=(23,))


# ---- 2-D
@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("pre", [oracle.FULL, oracle.POLYNOMIAL])
@pytest.mark.parametrize("N,bs", [((70, 45), None), ((70, 45), (40, 24)), ((3, 5), None)])
def test_warp2_gather_fp64(m, pre, N, bs):
    kw = {"blockSize": bs} if bs else {}
    check("forward", N, 50001, m, F64, pre, ["gather_warp2_kernel"], **kw)


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("pre", [oracle.FULL, oracle.POLYNOMIAL])
def test_warp2_gather_fp32(m, pre):
    check("forward", (70, 45), 15001, m, F32, pre, ["gather_warp2_kernel"])


@pytest.mark.parametrize("m", [2, 3, 4])
@pytest.mark.parametrize("pre", [oracle.FULL, oracle.POLYNOMIAL])
@pytest.mark.parametrize("N,bs", [((70, 45), None), ((70, 45), (40, 24)), ((3, 5), None)])
def test_warp2_spread_fp64(m, pre, N, bs):
    kw = {"blockSize": bs} if bs else {}
    check("adjoint", N, 9001, m, F64, pre, ["spread_warp2_kernel"], **kw)


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("dtype", [F32, F64])
def test_warp2_columns(m, dtype):
    """Stacks (table windows): both directions through the one-warp kernels, each column as a single plan's."""
    N, M, C = (40, 36), 6000, 8
    k = nodes(2, M, dtype, 577, m)
    rng = np.random.default_rng(m)
    p = nf.plan_nfft(k, N + (C,), dims=(1, 2), m=m, sigma=2.0)
    f = nf.as_colmajor(rng.standard_normal(N + (C,)) + 1j * rng.standard_normal(N + (C,)), N + (C,), p.cdtype)
    v = nf.as_colmajor(rng.standard_normal((M, C)) + 1j * rng.standard_normal((M, C)), (M, C), p.cdtype)
    y, x = nf.empty_image((M, C), p.cdtype), nf.empty_image(N + (C,), p.cdtype)
    fwd, adj = (lambda: nf.mul_(y, p, f)), (lambda: nf.mul_(x, nf.adjoint(p), v))
    fwd(), adj()
    assert launched(fwd, "gather_warp2_kernel") and launched(adj, "spread_warp2_kernel")
    fwd(), adj()
    one = nf.plan_nfft(k, N, m=m, sigma=2.0, precompute=nf.LINEAR)
    tol = 1e-5 if dtype == F32 else 1e-11
    for c in range(C):
        fc, vc = nf.as_colmajor(f[:, :, c], N, p.cdtype), v[:, c].contiguous()
        assert oracle.rel_l2(y[:, c].cpu().numpy(), (one * fc).cpu().numpy()) < tol
        assert oracle.rel_l2(x[:, :, c].cpu().numpy(), (nf.adjoint(one) * vc).cpu().numpy()) < tol


@pytest.mark.parametrize("m", [2, 3, 5, 6, 7, 8])
@pytest.mark.parametrize("pre", [nf.TENSOR, nf.POLYNOMIAL])
def test_batch_fp32_widths(m, pre):
    """Members of uneven sizes equal their own transforms (1e-6, as in the batch tests at m = 4)."""
    shapes, Ms = [(64, 64), (100, 36), (33, 31)], [20000, 700, 5000]
    rng = np.random.default_rng(m)
    plans = [nf.plan_nfft(nodes(2, M, F32, M // 3, i), N, m=m, sigma=2.0, precompute=pre)
             for i, (N, M) in enumerate(zip(shapes, Ms))]
    fs = [nf.as_colmajor(rng.standard_normal(N) + 1j * rng.standard_normal(N), N, torch.complex64) for N in shapes]
    vs = [torch.as_tensor(rng.standard_normal(M) + 1j * rng.standard_normal(M)).to("cuda", torch.complex64) for M in Ms]
    batch = nf.NFFTBatch(plans)
    for p, f, v, y, x in zip(plans, fs, vs, batch.forward(fs), batch.adjoint(vs)):
        assert oracle.rel_l2(y.cpu().numpy(), (p * f).cpu().numpy()) <= 1e-6
        assert oracle.rel_l2(x.cpu().numpy(), (nf.adjoint(p) * v).cpu().numpy()) <= 1e-6


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("pre", [nf.TENSOR, nf.FULL, nf.LINEAR])
def test_tiled_node_gradient_fp64(m, pre):
    """Against the plain path: the same window values and derivatives in another order, 1e-11."""
    N, M = (40, 27), 33001
    k = nodes(2, M, F64, 333, m)
    rng = np.random.default_rng(m)
    f = nf.as_colmajor(rng.standard_normal(N) + 1j * rng.standard_normal(N), N, torch.complex128)
    w = torch.as_tensor(rng.standard_normal(M) + 1j * rng.standard_normal(M)).cuda()
    out = []
    for kw in ({}, {"blocking": False}):
        p = nf.plan_nfft(k, N, m=m, sigma=2.0, precompute=pre, **kw)
        dk = torch.empty((M, 2), dtype=torch.float64, device="cuda")
        call = lambda: p.grad_nodes_(dk.t(), f, w)  # noqa: E731
        call()
        assert kw or launched(call, "grad_warp2_kernel")
        call()
        out.append(dk.cpu().numpy())
    assert oracle.rel_l2(out[0], out[1]) < 1e-11


# ---- 3-D
@pytest.mark.parametrize("m", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("pre", TABLES)
@pytest.mark.parametrize("bs", [(16, 8, 8), (8, 8, 8)])
@pytest.mark.parametrize("N", [(48, 40, 36), (33, 29, 31), (10, 9, 8)])
def test_plane3_gather(m, pre, bs, N):
    """Tiles inside the grid (bulk copies), tiles that wrap in every dimension, boxes larger than the grid."""
    kernels = ["gather_plane3_kernel"] + (["interp_tile3_kernel"] if m == 4 and N[0] == 48 else [])
    check("forward", N, 140001 if m == 2 else 100001, m, F32, pre, kernels, blockSize=bs)


@pytest.mark.parametrize("pre", TABLES)
@pytest.mark.parametrize("bs", [(16, 8, 8), (8, 8, 8), (16, 16, 8), (32, 8, 8)])
def test_tile3_gather(pre, bs):
    check("forward", (80, 72, 64), 150001, 4, F32, pre, ["interp_tile3_kernel"], blockSize=bs)


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("pre", [oracle.FULL, oracle.POLYNOMIAL])
@pytest.mark.parametrize("bs", [(16, 8, 4), (8, 8, 8), (5, 7, 3)])
def test_double3_gather(m, pre, bs):
    check("forward", (23, 17, 20), 70001, m, F64, pre, ["gather_double3_kernel"], blockSize=bs)


@pytest.mark.parametrize("m", [2, 3, 5])
@pytest.mark.parametrize("pre", [oracle.FULL, oracle.POLYNOMIAL])
@pytest.mark.parametrize("N,bs", [((36, 34, 40), None), ((23, 17, 20), (5, 7, 3)), ((40, 44, 30), (8, 8, 4))])
def test_double3_spread(m, pre, N, bs):
    kw = {"blockSize": bs} if bs else {}
    check("adjoint", N, 30001, m, F64, pre, ["spread_double3_kernel"], **kw)

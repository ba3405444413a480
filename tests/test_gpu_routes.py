"""Which kernel a call takes on both sides of the rules of dispatch, and that its
values agree with the oracle there: 1e-5 (FP32), 1e-11 (FP64; 1e-10 for polynomial
windows with m >= 6, the conditioning of two fits of degree 2m).

Each rule lies where the times of both kernels, beside it in the source, cross."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402
from kernel_route import launched  # noqa: E402
from oracle import oracle  # noqa: E402

ALL = ("spread_line_kernel", "spread_line_kahan_kernel", "spread_pad1_kernel", "gather_line_kernel", "gather_lanes_kernel",
       "interp_kernel",
       "gather_warp2_kernel", "gather_plane3_kernel", "gather_double3_kernel", "interp_tile3_kernel",
       "spread_warp2_kernel", "spread_owned_kernel", "spread_plane3_kernel", "spread_double3_kernel",
       "grad_nodes_kernel", "grad_warp2_kernel")
F32, F64 = np.float32, np.float64

# direction, N, M, m, precision, plan keywords, kernel
ROWS = [
    # 1-D spreading: tiles of 8 cells (grids of 512 and 8,000 points), 32 cells, 512 cells
    ("adjoint", (256,), 70000, 3, F32, {"compensated": True}, "spread_line_kernel"),
    ("adjoint", (4000,), 70000, 3, F32, {"compensated": True}, "spread_line_kahan_kernel"),
    ("adjoint", (16384,), 70000, 5, F32, {"compensated": True}, "spread_line_kahan_kernel"),
    ("adjoint", (16384,), 130000, 5, F32, {"compensated": True}, "spread_line_kernel"),
    ("adjoint", (40000,), 130000, 5, F32, {"compensated": True, "blockSize": (512,)}, "spread_line_kernel"),
    ("adjoint", (4000,), 130000, 4, F64, {"compensated": True}, "spread_line_kahan_kernel"),
    ("adjoint", (256,), 70000, 6, F32, {}, "spread_line_kernel"),
    ("adjoint", (4000,), 70000, 6, F32, {}, "spread_pad1_kernel"),
    ("adjoint", (4000,), 140000, 8, F32, {}, "spread_line_kernel"),
    ("adjoint", (128,), 70000, 3, F64, {}, "spread_pad1_kernel"),
    ("adjoint", (4000,), 140000, 3, F64, {}, "spread_line_kernel"),
    ("adjoint", (16384,), 130000, 4, F64, {}, "spread_pad1_kernel"),
    # 3-D gather, m = 4: 2048 and 4000 tasks
    ("forward", (64, 64, 64), 38000, 4, F32, {}, "interp_kernel"),
    ("forward", (64, 64, 64), 43000, 4, F32, {}, "interp_tile3_kernel"),
    ("forward", (80, 80, 80), 48000, 4, F32, {}, "interp_kernel"),
    ("forward", (80, 80, 80), 56000, 4, F32, {}, "interp_tile3_kernel"),
    # 1-D gather
    ("forward", (128,), 1000, 8, F64, {"precompute": oracle.POLYNOMIAL}, "gather_lanes_kernel"),
    ("forward", (20000,), 6143, 5, F64, {"precompute": oracle.POLYNOMIAL}, "gather_lanes_kernel"),
    ("forward", (3,), 33, 7, F64, {"precompute": oracle.POLYNOMIAL}, "gather_lanes_kernel"),
    ("forward", (500,), 1, 6, F64, {"precompute": oracle.POLYNOMIAL, "compensated": True}, "gather_lanes_kernel"),
    ("forward", (20000,), 6144, 5, F64, {"precompute": oracle.POLYNOMIAL}, "gather_line_kernel"),
    ("forward", (128,), 1000, 8, F64, {}, "gather_line_kernel"),
    ("forward", (128,), 1000, 4, F64, {"precompute": oracle.POLYNOMIAL}, "gather_line_kernel"),
    ("forward", (128,), 32000, 8, F32, {}, "gather_line_kernel"),
    # 3-D FP64 spreading: tiles of 8 x 8 x 4 (1024 tasks) and 5 x 7 x 3
    ("adjoint", (32, 32, 32), 14000, 5, F64, {}, "spread_owned_kernel"),
    ("adjoint", (32, 32, 32), 17000, 5, F64, {}, "spread_double3_kernel"),
    ("adjoint", (32, 32, 32), 14000, 3, F64, {}, "spread_double3_kernel"),
    ("adjoint", (32, 32, 32), 17000, 7, F64, {}, "spread_owned_kernel"),
    ("adjoint", (23, 17, 20), 4000, 6, F64, {"blockSize": (5, 7, 3), "precompute": oracle.FULL}, "spread_owned_kernel"),
    # 2-D gathers of a single plan
    ("forward", (44, 44), 14335, 5, F32, {}, "interp_kernel"),
    ("forward", (44, 44), 14336, 5, F32, {}, "gather_warp2_kernel"),
    ("forward", (44, 44), 14337, 3, F32, {"precompute": oracle.POLYNOMIAL}, "gather_warp2_kernel"),
    ("forward", (44, 44), 10239, 8, F32, {"precompute": oracle.FULL}, "interp_kernel"),
    ("forward", (44, 44), 10240, 8, F32, {"precompute": oracle.FULL}, "gather_warp2_kernel"),
    ("forward", (128, 128), 16384, 4, F64, {}, "gather_warp2_kernel"),
    ("forward", (128, 128), 16383, 4, F64, {}, "interp_kernel"),
    ("forward", (128, 128), 49151, 5, F64, {}, "interp_kernel"),
    ("forward", (128, 128), 49152, 5, F64, {}, "gather_warp2_kernel"),
]


@pytest.mark.parametrize("row", range(len(ROWS)))
def test_route_and_values(row):
    direction, N, M, m, dtype, kw, kernel = ROWS[row]
    rng = np.random.default_rng(row)
    k = (rng.random((len(N), M)) - 0.5).astype(dtype)
    kw = dict(kw)
    pre = kw.pop("precompute", oracle.TENSOR)
    f = (rng.standard_normal(N) + 1j * rng.standard_normal(N)).astype(np.complex64)
    v = (rng.standard_normal(M) + 1j * rng.standard_normal(M)).astype(np.complex64)
    p = nf.plan_nfft(k, N, m=m, sigma=2.0, precompute=pre, **kw)
    op = oracle.OraclePlan(k.astype(np.float64), N, m=m, sigma=2.0, precompute=pre)
    tol = 1e-5 if dtype == F32 else (1e-10 if pre != oracle.FULL and m >= 6 else 1e-11)
    fd, vd = nf.as_colmajor(f, N, p.cdtype), torch.as_tensor(v).to(device="cuda", dtype=p.cdtype)
    if direction == "forward":
        y = torch.empty_like(vd)
        call, got, ref = (lambda: nf.mul_(y, p, fd)), y, op.forward(f.astype(np.complex128))
    else:
        x = nf.empty_image(N, p.cdtype)
        call, got, ref = (lambda: nf.mul_(x, nf.adjoint(p), vd)), x, op.adjoint(v.astype(np.complex128))
    call()
    assert launched(call, *ALL) == {kernel}
    call()
    assert oracle.rel_l2(got.cpu().numpy().ravel(order="F"), ref.ravel(order="F")) < tol


@pytest.mark.parametrize("m,M,C,kernel", [(4, 900, 2, "spread_owned_kernel"), (4, 9000, 3, "spread_warp2_kernel"),
                                          (5, 6000, 4, "spread_owned_kernel"), (5, 6000, 8, "spread_warp2_kernel"),
                                          (7, 3000, 20, "spread_owned_kernel"), (7, 6000, 8, "spread_warp2_kernel"),
                                          (8, 9000, 5, "spread_owned_kernel")])
def test_fp64_stack(m, M, C, kernel):
    """FP64 directional plans: one or two warps per tile; each column equals its single 2-D plan."""
    N = (40, 36)
    rng = np.random.default_rng(m)
    k = rng.random((2, M)) - 0.5
    v = nf.as_colmajor(rng.standard_normal((M, C)) + 1j * rng.standard_normal((M, C)), (M, C), torch.complex128)
    p = nf.plan_nfft(k, N + (C,), dims=(1, 2), m=m, sigma=2.0)
    x = nf.empty_image(N + (C,), torch.complex128)
    nf.mul_(x, nf.adjoint(p), v)
    assert launched(lambda: nf.mul_(x, nf.adjoint(p), v), *ALL) == {kernel}
    nf.mul_(x, nf.adjoint(p), v)
    one = nf.plan_nfft(k, N, m=m, sigma=2.0, precompute=nf.LINEAR)
    for c in range(C):
        assert oracle.rel_l2(x[:, :, c].cpu().numpy(), (nf.adjoint(one) * v[:, c].contiguous()).cpu().numpy()) < 1e-11


@pytest.mark.parametrize("m", [3, 5, 7, 8])
@pytest.mark.parametrize("pre", [nf.TENSOR, nf.POLYNOMIAL])
@pytest.mark.parametrize("Ms", [(2500, 700, 1900), (30000, 9000, 4000, 0), (60000,) * 9])
def test_fp64_batch(m, pre, Ms):
    """FP64 batches of few, some and many nodes: every member equals its own transforms (1e-12, as in the batch tests)."""
    rng = np.random.default_rng(len(Ms) + m)
    shapes = [((64, 48), (33, 31), (96, 20), (40, 40))[i % 4] for i in range(len(Ms))]
    plans = [nf.plan_nfft(rng.random((2, M)) - 0.5, N, m=m, sigma=2.0, precompute=pre) for N, M in zip(shapes, Ms)]
    fs = [nf.as_colmajor(rng.standard_normal(N) + 1j * rng.standard_normal(N), N, torch.complex128) for N in shapes]
    vs = [torch.as_tensor(rng.standard_normal(M) + 1j * rng.standard_normal(M)).cuda() for M in Ms]
    y1 = [(p * f).cpu().numpy() for p, f in zip(plans, fs)]
    x1 = [(nf.adjoint(p) * v).cpu().numpy() for p, v in zip(plans, vs)]
    batch = nf.NFFTBatch(plans)
    for _ in range(2):
        for i, (y, x) in enumerate(zip(batch.forward(fs), batch.adjoint(vs))):
            if Ms[i]:
                assert oracle.rel_l2(y.cpu().numpy(), y1[i]) <= 1e-12
            assert oracle.rel_l2(x.cpu().numpy(), x1[i]) <= 1e-12 if Ms[i] else bool((x == 0).all())


@pytest.mark.parametrize("m,M,pre,dtype,kernel", [(4, 9000, nf.TENSOR, F64, "grad_nodes_kernel"),
                                                  (4, 13000, nf.TENSOR, F64, "grad_warp2_kernel"),
                                                  (8, 13000, nf.LINEAR, F64, "grad_warp2_kernel"),
                                                  (5, 13000, nf.FULL, F64, "grad_nodes_kernel"),
                                                  (5, 17000, nf.FULL, F64, "grad_warp2_kernel"),
                                                  (8, 30000, nf.FULL, F64, "grad_nodes_kernel"),
                                                  (8, 33000, nf.FULL, F64, "grad_warp2_kernel"),
                                                  (8, 3000, nf.FULL, F32, "grad_warp2_kernel")])
def test_node_gradient(m, M, pre, dtype, kernel):
    """By tiles or a warp per node; against the plain path (5e-5 / 1e-11, as in the node gradient's tests)."""
    N = (40, 27)
    rng = np.random.default_rng(m)
    k = (rng.random((2, M)) - 0.5).astype(dtype)
    f = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    w = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    out = []
    for kw in ({}, {"blocking": False}):
        p = nf.plan_nfft(k, N, m=m, sigma=2.0, precompute=pre, **kw)
        fd, wd = nf.as_colmajor(f, N, p.cdtype), torch.as_tensor(w).to(device="cuda", dtype=p.cdtype)
        dk = torch.empty((M, 2), dtype=p.dtype, device="cuda")
        call = lambda: p.grad_nodes_(dk.t(), fd, wd)  # noqa: E731
        call()
        if not kw:
            assert launched(call, *ALL) == {kernel}
            call()
        out.append(dk.cpu().numpy())
    assert oracle.rel_l2(out[0], out[1]) < (5e-5 if dtype == F32 else 1e-11)

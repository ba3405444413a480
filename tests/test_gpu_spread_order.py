"""Successive nodes that share tile points across lanes: every spreader that adds
into a shared-memory tile without atomics.

600 nodes walk one grid cell at a time (along x, y, z and diagonally, and on the
spot), so that a point written for one node is read by another lane for the next;
an update lost between lanes shows in the sums.  Against the oracle, 1e-5 (FP32)
and 1e-11 (FP64), the suite's bars; each case asserts which kernel ran."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402
from kernel_route import launched  # noqa: E402
from oracle import oracle  # noqa: E402

CASES = [  # D, N, M, m, FP64, plan keywords, environment, kernel
    (2, (48, 40), 6000, 3, False, {}, {}, "spread_warp2_kernel"),
    (2, (48, 40), 6000, 4, False, {}, {}, "spread_warp2_kernel"),
    (2, (48, 40), 6000, 8, False, {}, {}, "spread_warp2_kernel"),
    (2, (48, 40), 6000, 4, True, {}, {}, "spread_warp2_kernel"),
    (2, (48, 40), 6000, 5, True, {}, {}, "spread_owned_kernel"),
    (2, (48, 40), 6000, 4, False, {"compensated": True}, {}, "spread_owned_kernel"),
    (3, (40, 36, 32), 6000, 2, False, {}, {}, "spread_plane3_kernel"),
    (3, (40, 36, 32), 6000, 4, False, {}, {}, "spread_plane3_kernel"),
    (3, (40, 36, 32), 6000, 5, False, {}, {}, "spread_plane3_kernel"),
    (3, (40, 36, 32), 6000, 4, False, {}, {"NFFT_GB300_SPREAD_REC": "0"}, "spread_tile3_kernel"),
    (3, (40, 36, 32), 6000, 5, False, {}, {"NFFT_GB300_SPREAD_REC": "0"}, "spread_owned_kernel"),
    (3, (23, 17, 20), 9000, 3, True, {"blockSize": (5, 7, 3)}, {}, "spread_double3_kernel"),
    (3, (23, 17, 20), 9000, 5, True, {"blockSize": (5, 7, 3)}, {}, "spread_owned_kernel"),  # few nodes per tile
    (3, (23, 17, 20), 9000, 4, True, {"blockSize": (5, 7, 3)}, {}, "spread_owned_kernel"),
    (3, (23, 17, 20), 13000, 5, True, {"blockSize": (5, 7, 3)}, {}, "spread_double3_kernel"),
]
KERNELS = ("spread_warp2_kernel", "spread_owned_kernel", "spread_plane3_kernel", "spread_tile3_kernel",
           "spread_double3_kernel")


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("pre", [oracle.TENSOR, oracle.POLYNOMIAL])
def test_neighbouring_nodes(monkeypatch, case, pre):
    D, N, M, m, double, kw, env, kernel = CASES[case]
    for key, value in env.items():
        monkeypatch.setenv(key, value)
    rng = np.random.default_rng(case)
    k = rng.random((D, M)) - 0.5
    cell = 1.0 / (2 * np.array(N))
    i = np.arange(600)
    step = np.stack([(i // 4 + (i % 5 == d)) % 6 for d in range(D)])  # a diagonal walk with single steps in each dimension
    step[:, 400:] = 0                                                # and nodes on the spot
    k[:, 100:700] = 0.05 + cell[:, None] * (step + 0.3 * rng.random((D, 600)))
    dtype = np.float64 if double else np.float32
    k = k.astype(dtype)
    v = (rng.standard_normal(M) + 1j * rng.standard_normal(M)).astype(np.complex64)
    p = nf.plan_nfft(k, N, m=m, sigma=2.0, precompute=pre, **kw)
    x = torch.as_tensor(v).to(device="cuda", dtype=p.cdtype)
    f = nf.empty_image(N, p.cdtype)
    nf.mul_(f, nf.adjoint(p), x)
    assert launched(lambda: nf.mul_(f, nf.adjoint(p), x), *KERNELS) == {kernel}
    op = oracle.OraclePlan(k.astype(np.float64), N, m=m, sigma=2.0, precompute=pre)
    ref = op.adjoint(v.astype(np.complex128))
    for _ in range(5):
        nf.mul_(f, nf.adjoint(p), x)
        assert oracle.rel_l2(f.cpu().numpy().ravel(order="F"), ref.ravel(order="F")) < (1e-11 if double else 1e-5)

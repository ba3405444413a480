"""The 3-D FP32 plane-owner spreader and the tiled gather (spread_plane3.cuh,
gather3.cu) for every window width they are compiled for, against the oracle.

Both tile shapes, table and polynomial windows, tiles inside the grid (bulk
tensor copies and reductions) and tiles that wrap in every dimension, a grid
that is no whole number of tiles, a hot tile of several batches with a
remainder, tiles without the bulk copies, and node sets too sparse for the
tiled gather.  Tolerance: the suite's FP32 parity bar, 1e-5."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402
from oracle import oracle  # noqa: E402

TOL32 = 1e-5


def problem(N, M, seed):
    rng = np.random.default_rng(seed)
    k = (rng.random((3, M)) - 0.5).astype(np.float32)
    k[:, :5] = np.array([[-0.5, 0.4999, 0.0, -0.001, 0.25]] * 3, dtype=np.float32)
    if M > 2000:
        k[:, 50:50 + 181] = 0.2 + 0.002 * rng.random((3, 181)).astype(np.float32)
    f = (rng.standard_normal(N) + 1j * rng.standard_normal(N)).astype(np.complex64)
    v = (rng.standard_normal(M) + 1j * rng.standard_normal(M)).astype(np.complex64)
    return k, f, v


def check(N, M, m, pre, bs, seed=3):
    k, f, v = problem(N, M, seed)
    p = nf.plan_nfft(k, N, m=m, sigma=2.0, precompute=pre, blockSize=bs)
    op = oracle.OraclePlan(k.astype(np.float64), N, m=m, sigma=2.0, precompute=pre)
    y = (p * nf.as_colmajor(f, N, torch.complex64)).cpu().numpy()
    x = (nf.adjoint(p) * torch.as_tensor(v)).cpu().numpy()
    assert oracle.rel_l2(y, op.forward(f.astype(np.complex128))) < TOL32
    assert oracle.rel_l2(x.ravel(order="F"), op.adjoint(v.astype(np.complex128)).ravel(order="F")) < TOL32
    assert nf.load().nfft_sync(p._handle) == 0


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("pre", [oracle.TENSOR, oracle.POLYNOMIAL])
@pytest.mark.parametrize("bs", [(16, 8, 8), (8, 8, 8)])
@pytest.mark.parametrize("N", [(48, 40, 36), (33, 29, 31)])
def test_plane3_matches_oracle(m, pre, bs, N):
    check(N, 9000, m, pre, bs)


@pytest.mark.parametrize("m", [3, 5])
def test_plane3_without_bulk_copies(monkeypatch, m):
    monkeypatch.setenv("NFFT_GB300_SPREAD_TMA", "0")
    monkeypatch.setenv("NFFT_GB300_SPREAD_ZERO_COPY", "0")
    check((48, 40, 36), 9000, m, oracle.TENSOR, (16, 8, 8))


@pytest.mark.parametrize("m", [2, 3, 5, 6])
def test_plane3_sparse_and_tiny(m):
    check((40, 40, 40), 61, m, oracle.POLYNOMIAL, (16, 8, 8))   # fewer than six nodes per task
    check((10, 9, 8), 1500, m, oracle.TENSOR, (8, 8, 8))         # every tile wraps, boxes exceed the grid


@pytest.mark.parametrize("m", [3, 4, 5])
def test_first_adjoint_inside_a_capture(m):
    """The first adjoint of a plan, captured into a graph by the caller: nothing is allocated for it."""
    N = (48, 40, 32)
    k, _, v = problem(N, 3000, 7)
    want = (nf.adjoint(nf.plan_nfft(k, N, m=m, sigma=2.0)) * torch.as_tensor(v)).cpu().numpy()
    p = nf.plan_nfft(k, N, m=m, sigma=2.0)
    x = torch.as_tensor(v).cuda()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = nf.adjoint(p) * x
    for _ in range(2):
        graph.replay()
        torch.cuda.synchronize()
        assert oracle.rel_l2(y.cpu().numpy().ravel(), want.ravel()) < TOL32
    y = (nf.adjoint(p) * x).cpu().numpy()  # and outside one
    assert oracle.rel_l2(y.ravel(), want.ravel()) < TOL32


@pytest.mark.parametrize("m,M", [(3, 140001), (4, 3 * 2**20 + 7), (5, 3 * 2**20 + 7)])
@pytest.mark.parametrize("pre", [oracle.TENSOR, oracle.POLYNOMIAL])
def test_many_nodes(m, M, pre):
    """Two warps per tile (node sets beyond the rule's lines), against the same adjoint in double precision."""
    N = (40, 36, 44)
    k, _, v = problem(N, M, 11)
    x = (nf.adjoint(nf.plan_nfft(k, N, m=m, sigma=2.0, precompute=pre)) * torch.as_tensor(v)).cpu().numpy()
    q = nf.plan_nfft(k.astype(np.float64), N, m=m, sigma=2.0, precompute=pre)
    y = (nf.adjoint(q) * torch.as_tensor(v.astype(np.complex128))).cpu().numpy()
    assert oracle.rel_l2(x.ravel(), y.ravel()) < TOL32

"""The node binning of nodes! (sort.cu, precompute.cu) at its own edges: node
counts around a warp, a sort CTA (1024 and 4096 keys) and the switch between
them (2^20), tile counts around the one-CTA tile lists (8192), key widths of one
to three passes; permutation and tile starts are compared bit for bit with
numpy's stable sort of the tile index.  Rejected nodes (out of range, NaN,
infinite) raise and leave the plan ready for the next nodes!."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402


def expected(k, Nt, bs):
    """Tile of every node: shift to [0, 1), truncate, divide by the tile (dimension 1 fastest)."""
    t = np.zeros(k.shape[1], np.int64)
    stride = 1
    for d in range(k.shape[0]):
        x = k[d].copy()
        x = np.where(x < 0, x + k.dtype.type(1), x)
        x = np.where(x == 1, x - np.finfo(k.dtype).eps, x).astype(k.dtype)
        g = np.clip((x * k.dtype.type(Nt[d])).astype(np.int64), 0, Nt[d] - 1)
        t += stride * (g // bs[d])
        stride *= -(-Nt[d] // bs[d])
    perm = np.argsort(t, kind="stable").astype(np.int32)
    return perm, np.concatenate([[0], np.cumsum(np.bincount(t, minlength=stride))]).astype(np.int32)


@pytest.mark.parametrize("M", [1, 31, 33, 1023, 1025, 4097, 70001, (1 << 20) - 1, 1 << 20, (1 << 20) + 5])
@pytest.mark.parametrize("N,bs", [((64, 64), (64, 64)), ((64, 64), (16, 8)), ((512, 512), (8, 16)),
                                  ((513, 512), (8, 16)), ((64, 60, 58), (8, 8, 8))])
def test_binning_edges(M, N, bs):
    rng = np.random.default_rng(M)
    k = (rng.random((len(N), M)) - 0.5).astype(np.float32)
    if M > 100:
        k[:, M // 3:M // 2] *= np.float32(0.01)  # hot tiles
    p = nf.plan_nfft(k, N, m=2, sigma=2.0, blockSize=bs)
    b = p.binning()
    perm, start = expected(k, p.Ntilde, bs)
    assert np.array_equal(b["perm"], perm)
    assert np.array_equal(b["tile_start"], start)


@pytest.mark.parametrize("bad", [0.51, -0.6, 1e30, np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("pre", ["FULL", "LINEAR", "POLYNOMIAL"])
def test_rejected_nodes_leave_the_plan_usable(bad, dtype, pre):
    rng = np.random.default_rng(1)
    N, M = (20, 24), 900
    k = (rng.random((2, M)) - 0.5).astype(dtype)
    f = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    p = nf.plan_nfft(k, N, m=4, sigma=2.0, precompute=getattr(nf, pre))
    y = (p * nf.as_colmajor(f, N, p.cdtype)).cpu().numpy()
    wrong = k.copy()
    wrong[1, 777] = bad
    with pytest.raises(nf.ArgumentError):
        p.nodes_(wrong)
    p.nodes_(k)
    assert np.array_equal((p * nf.as_colmajor(f, N, p.cdtype)).cpu().numpy(), y)

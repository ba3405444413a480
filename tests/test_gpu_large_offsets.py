"""Long 3-D grids: tap offsets of the tiled FP32 gather where a tile plane times
the node's z index passes 2^31 (grids of more than about 4 million planes).

The nodes lie in the tiles on both sides of that index; the tiled gather (one
point per copy and per-task tiles) against the direct one, which forms 64-bit grid
offsets.  Both sum (2m)^3 = 1728 products in FP32 in another order: 1e-5, the
suite's FP32 bar."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402
from kernel_route import launched  # noqa: E402
from oracle import oracle  # noqa: E402


def test_tiled_gather_beyond_2p31_tile_offsets(monkeypatch):
    N, m, M = (4, 4, 2100000), 6, 40000
    plane = 28 * 19                       # tile plane of an 8 x 8 tile, 12 taps: row pitch x rows
    z = 2**31 // plane - 140              # about 35 tiles of 8 planes around the index
    rng = np.random.default_rng(5)
    k = rng.random((3, M)) - 0.5
    k[2] = (z + 280 * rng.random(M)) / (2 * N[2]) - 1.0
    k = k.astype(np.float32)
    p = nf.plan_nfft(k, N, m=m, sigma=2.0, blockSize=(8, 8, 8))
    assert p.Ntilde == (8, 8, 2 * N[2])
    g = nf.empty_image(p.Ntilde, torch.complex64)
    g.copy_(torch.randn(p.Ntilde[::-1], dtype=torch.complex64, device="cuda").permute(2, 1, 0))
    y = torch.empty(M, dtype=torch.complex64, device="cuda")
    assert launched(lambda: p.convolve_(g, y), "gather_plane3_kernel")
    p.convolve_(g, y)
    assert nf.load().nfft_sync(p._handle) == 0
    del p
    monkeypatch.setenv("NFFT_GB300_GATHER_TMA", "0")
    q = nf.plan_nfft(k, N, m=m, sigma=2.0, blockSize=(8, 8, 8))
    ref = torch.empty_like(y)
    q.convolve_(g, ref)
    assert oracle.rel_l2(y.cpu().numpy(), ref.cpu().numpy()) < 1e-5

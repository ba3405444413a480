"""Line FFTs with few lines per CTA (small transforms, fft.cu): every supported
length in both precisions, image sizes that leave a last CTA partly empty, 2-D
and 3-D, against the oracle.  Tolerances: the suite's parity bars, 1e-11 (FP64)
and 1e-5 (FP32)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402
from oracle import oracle  # noqa: E402


# (N, sigma): every Ntilde = 2 (ceil(sigma N) div 2) is a power of two; odd and ragged N included
CASES = [((32, 32), 2.0), ((64, 32), 2.0), ((128, 64), 2.0), ((256, 256), 2.0), ((512, 32), 2.0), ((32, 512), 2.0),
         ((64, 32, 32), 2.0), ((51, 51), 1.26), ((205, 205), 1.25), ((43, 43, 43), 1.5)]


@pytest.mark.parametrize("N,sigma", CASES)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_small_fused_transforms(N, sigma, dtype):
    rng = np.random.default_rng(sum(N))
    D, M = len(N), 700
    k = (rng.random((D, M)) - 0.5).astype(dtype)
    f = (rng.standard_normal(N) + 1j * rng.standard_normal(N)).astype(np.complex64)
    v = (rng.standard_normal(M) + 1j * rng.standard_normal(M)).astype(np.complex64)
    p = nf.plan_nfft(k, N, m=4, sigma=sigma)
    assert all(n & (n - 1) == 0 for n in p.Ntilde)
    op = oracle.OraclePlan(k.astype(np.float64), N, m=4, sigma=sigma, precompute=oracle.POLYNOMIAL)
    tol = 1e-5 if dtype == np.float32 else 1e-11
    y = (p * nf.as_colmajor(f, N, p.cdtype)).cpu().numpy()
    x = (nf.adjoint(p) * torch.as_tensor(v).to(p.cdtype)).cpu().numpy()
    assert oracle.rel_l2(y, op.forward(f.astype(np.complex128))) < tol
    assert oracle.rel_l2(x.ravel(order="F"), op.adjoint(v.astype(np.complex128)).ravel(order="F")) < tol

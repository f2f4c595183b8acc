"""SIMT GEMM at the edges of its tile rule: batches of 64 x 64 and of 32 x 32 tiles
(complex64), of whole 32 x 32 ones (complex128), inner dimensions around the K-steps
of 8, 16 and 32.  Bound of test_simt_tiles.py: a sum of K products is within 2 K u of
the sum of magnitudes, twice that against a reference of the same rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from atlasq_gb300 import ops  # noqa: E402

DEV = "cuda:0"


@pytest.mark.parametrize("K", [1, 7, 8, 9, 15, 17, 33])
@pytest.mark.parametrize("M,N,batch", [(33, 34, 160), (64, 64, 152), (65, 64, 80), (5, 7, 310), (31, 70, 110),
                                       (32, 64, 800), (32, 32, 1520)])
@pytest.mark.parametrize("dt", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("opA,opB", [("N", "N"), ("C", "T")])
def test_batches(M, N, K, batch, dt, opA, opB):
    g = torch.Generator().manual_seed(M + N + K + batch)
    A = torch.randn(batch, *((M, K) if opA == "N" else (K, M)), generator=g, dtype=dt)
    B = torch.randn(batch, *((K, N) if opB == "N" else (N, K)), generator=g, dtype=dt)
    got = ops.cgemm(A.to(DEV), B.to(DEV), opA, opB).cpu().to(torch.complex128)
    a, b = A.to(torch.complex128), B.to(torch.complex128)
    a, b = (a if opA == "N" else a.mH), (b if opB == "N" else b.mT)
    unit = 2.0 ** -24 if dt == torch.complex64 else 2.0 ** -53
    assert bool(((got - a @ b).abs() <= 4 * K * unit * (a.abs() @ b.abs())).all())

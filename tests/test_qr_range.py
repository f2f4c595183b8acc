"""Blocked QR of matrices whose column norms squared lie at either end of the
float32 range: no column is taken for zero.

Bounds of test_qr_blocked.py, 2 N u; at 2e-20 the squares of the entries are
subnormal, each rounded by 2^-150, so the norms squared of M entries of size s^2 are
exact to 2^-150 / s^2 only, which a reflector of each of the N columns adds."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from atlasq_gb300 import ops  # noqa: E402

DEV = "cuda:0"


@pytest.mark.parametrize("scale", [2e-20, 1e-19, 3e-19, 1e-17, 1e15, 1e17])
@pytest.mark.parametrize("M,N", [(128, 64), (64, 100), (512, 256), (600, 16)])
def test_qr_at_the_ends_of_the_range(M, N, scale):
    g = torch.Generator().manual_seed(M + N)
    A = torch.randn(M, N, generator=g, dtype=torch.complex128)
    A = (A * scale).to(torch.complex64)
    Q, R = ops.qr(A.to(DEV))
    Q, R, A = (t.cpu().to(torch.complex128).numpy() for t in (Q, R, A))
    A, R = A / scale, R / scale  # norms that 64 bits square without underflow
    u = 2.0 ** -24 + 2.0 ** -150 / min(scale * scale, 1.0)
    k = min(M, N)
    assert np.linalg.norm(Q @ R - A) <= 2 * N * u * np.linalg.norm(A)
    assert np.linalg.norm(Q.conj().T @ Q - np.eye(k)) <= 2 * N * u * np.sqrt(k)

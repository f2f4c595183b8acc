"""The blocked cluster QR at its edges: partial last panels, panels past the rank
of a wide matrix, one and several panels per CTA, one and two V buffers (large
complex128), both orders and both output forms.

Householder QR: ||A - QR|| <= c N u ||A|| and ||Q^H Q - I|| <= c N u with a small
constant (c = 2 here, Frobenius norms, sqrt(N) for the identity's norm); R's
diagonal is real with the sign opposite to the column's leading entry's real
part, so R's diagonal also equals LAPACK's within the backward error of a
well-conditioned matrix."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from atlasq_gb300 import ops  # noqa: E402

DEV = "cuda:0"


@pytest.mark.parametrize("M,N", [(64, 33), (128, 100), (129, 31), (255, 256), (512, 200), (512, 256), (300, 300),
                                 (200, 333), (96, 250), (640, 130), (1000, 48)])
@pytest.mark.parametrize("dt", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("trans", [False, True])
def test_qr_edges(M, N, dt, trans):
    g = torch.Generator().manual_seed(M + N)
    A = torch.complex(torch.randn(M, N, generator=g, dtype=torch.float64),
                      torch.randn(M, N, generator=g, dtype=torch.float64)).to(dt)
    if trans:
        Qt, Rt = ops.qr(A.T.contiguous().to(DEV), transA=True, trans_out=True)
        Q, R = Qt.T, Rt.T
    else:
        Q, R = ops.qr(A.to(DEV))
    Q, R, A = (t.cpu().to(torch.complex128).numpy() for t in (Q, R, A))
    u = 2.0 ** -24 if dt == torch.complex64 else 2.0 ** -53
    k = min(M, N)
    assert np.linalg.norm(Q @ R - A) <= 2 * N * u * np.linalg.norm(A)
    assert np.linalg.norm(Q.conj().T @ Q - np.eye(k)) <= 2 * N * u * np.sqrt(k)
    assert np.all(np.tril(R[:, :k], -1) == 0)
    d = np.diagonal(np.linalg.qr(A)[1])
    assert np.max(np.abs(np.diagonal(R) - d)) <= 2 * N * u * np.linalg.norm(A)

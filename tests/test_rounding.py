"""Size of the rounding errors of complex64 QR and of the register-resident
tridiagonalisation, against 64 bits over seeded matrices, in units of u = 2^-24.

The limits lie where square roots, divisions and the rank-2 update are each rounded
once or twice at the size of their result, as in LAPACK's steps; measured with the
reflector's reciprocals unrefined and four roundings an update (first), each
rounded once (second), and in the packed kernels these replaced (third):
||QR - A|| / ||A|| of 128 x 64                         4.18  3.78  3.87
rms eigenvalue error over lambda_0, n = 100            0.592 0.521 0.526
||V diag(w) V^H - H|| / ||H||, n = 100                 8.90  7.44  7.80"""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from atlasq_gb300 import ops  # noqa: E402

DEV, U = "cuda:0", 2.0 ** -24


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, dtype=torch.complex64)


def test_qr_rounding():
    g, err = torch.Generator().manual_seed(1), []
    for _ in range(60):
        A = _randn(g, 128, 64)
        Q, R = (t.cpu().to(torch.complex128) for t in ops.qr(A.to(DEV)))
        A = A.to(torch.complex128)
        err.append(float((Q @ R - A).norm() / A.norm()))
    assert sum(err) / len(err) <= 4.0 * U


def test_eigensolver_rounding():
    g, values, matrix, n = torch.Generator().manual_seed(2), [], [], 100
    for _ in range(10):
        X = _randn(g, 20, n, n)
        H = X.mH @ X / n
        H = (H + H.mH) / 2
        w, V = (t.cpu() for t in ops.heevd(H.to(DEV)))
        H, V, w = H.to(torch.complex128), V.to(torch.complex128), w.double()
        ref = torch.linalg.eigvalsh(H).flip(-1)
        values.append(float(((w - ref) / ref[:, :1]).pow(2).mean()))
        back = (V * w[:, None, :].to(V.dtype)) @ V.mH
        matrix.append(float(((back - H).norm(dim=(1, 2)) / H.norm(dim=(1, 2))).mean()))
    assert (sum(values) / len(values)) ** 0.5 <= 0.555 * U
    assert sum(matrix) / len(matrix) <= 8.2 * U

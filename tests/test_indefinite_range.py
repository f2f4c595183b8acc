"""Eigenvalues of Hermitian matrices that are no Gram matrices: a zero diagonal (then
nothing scales H), a diagonal far below the couplings, couplings far below the rest
(the pair of determinants of the count shrinks by any factor a step), at scales
from 1e-25 to 1e25.

Tolerance: Householder tridiagonalisation is backward stable, |dlambda| <= 2 n u ||H||;
bisection adds 2 eps + 4 eps of the Gershgorin interval, at most 3 ||H||:
(2 n + 36) u ||H||.  Residuals (scales whose inverse iterates stay in range):
the reduction's (8 n + 64) u ||H||, as in test_vector_phase.py."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from atlasq_gb300 import ops  # noqa: E402

DEV = "cuda:0"


def _matrix(kind, n, scale):
    g = torch.Generator().manual_seed(n)
    X = torch.randn(n, n, generator=g, dtype=torch.complex128)
    H = (X + X.mH) / 2
    if kind == "zero":
        H -= torch.diag_embed(torch.diagonal(H))
    elif kind == "tiny":
        H += torch.diag_embed((1e-8 * torch.rand(n, generator=g, dtype=torch.float64) - torch.diagonal(H).real)
                              .to(torch.complex128))
    elif kind == "path":  # already tridiagonal, zero diagonal
        H = torch.diag_embed(torch.ones(n - 1, dtype=torch.complex128), 1)
        H = H + H.mH
    elif kind == "ones":
        H = torch.ones(n, n, dtype=torch.complex128)
    elif kind == "faint":  # two blocks, one of them 1e-13 of the other with a zero diagonal
        k = n // 2
        H[:k, k:] = 0
        H[k:, :k] = 0
        H[:k, :k] *= 1e-13
        H[:k, :k] -= torch.diag_embed(torch.diagonal(H[:k, :k]))
    return H * scale


@pytest.mark.parametrize("dt", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n", [5, 24, 100])
@pytest.mark.parametrize("kind,scale", [("zero", s) for s in (1e-25, 1e-12, 1e-9, 1.0, 1e8, 1e12, 1e25)] +
                         [("path", s) for s in (1e-20, 1e-12, 1e-10, 1e10, 1e12)] +
                         [("tiny", 1.0), ("tiny", 1e-4), ("ones", 1.0), ("ones", 1e6), ("faint", 1.0), ("faint", 1e6)])
def test_eigenvalues_of_any_hermitian_matrix(kind, scale, n, dt):
    H = _matrix(kind, n, scale).to(dt)
    w, V = ops.heevd(H.to(DEV))
    w = w.cpu().double().numpy()
    H = H.to(torch.complex128).numpy()
    ref = np.linalg.eigvalsh(H)[::-1]
    size = np.abs(ref).max()
    u = 2.0 ** -24 if dt == torch.complex64 else 2.0 ** -53
    assert np.max(np.abs(w - ref)) <= (2 * n + 36) * u * size
    if kind == "zero" and 1e-9 <= scale <= 1e9:
        V = V.cpu().to(torch.complex128).numpy()
        assert np.linalg.norm(H @ V - V * w) <= (8 * n + 64) * u * size

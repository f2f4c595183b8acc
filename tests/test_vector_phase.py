"""The back-transformation with one and with two columns per warp, bisection and
inverse iteration at their chunk edges, and the split column norms of the rank
selection.

The two column counts do the same arithmetic per column, so a matrix alone (few
columns: one per warp) and among copies (two per warp), reduced by the same number
of CTAs, has to give the same eigenvectors bit for bit.

Norms: ||X||^2 is summed to double accuracy over a float32 contraction that rounds
each entry by at most (chiM + 4) u of the product of the magnitudes it sums
(u = 2^-24), and the kept sigma^2 of an untruncated gate add up to it within the
basis's n u."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from atlasq_gb300 import AdaptiveMPS, _lib, ops  # noqa: E402
from atlasq_gb300 import adaptive_mps as amod  # noqa: E402

DEV = "cuda:0"


@pytest.mark.parametrize("n,C,many", [(65, 0, 20), (129, 2, 12), (300, 4, 6), (700, 8, 2)])
def test_columns_per_warp(n, C, many):
    g = torch.Generator().manual_seed(n)
    X = torch.randn(n + 3, n, generator=g, dtype=torch.complex128)
    H = (X.mH @ X).to(torch.complex64).to(DEV)
    lib = _lib.load()
    if C:
        for count in (1, many):
            rc = lib.agb_set_tridiag_cluster(_lib.AGB_C64, n, count, C, 512)
            if rc == _lib.AGB_ERR_UNSUPPORTED:
                pytest.skip("the device does not schedule this cluster size")
            assert rc == 0
    try:
        w1, v1 = ops.heevd(H.unsqueeze(0))
        w2, v2 = ops.heevd(H.unsqueeze(0).expand(many, n, n).contiguous())
    finally:
        if C:
            for count in (1, many):
                assert lib.agb_set_tridiag_cluster(_lib.AGB_C64, n, count, 0, 512) == 0
    assert torch.equal(w1[0], w2[0])
    assert torch.equal(v1[0], v2[0])


@pytest.mark.parametrize("dt,batch", [(torch.complex64, 2), (torch.complex128, 2)])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 15, 16, 17, 18, 20, 32, 33, 47, 64, 65, 100])
def test_eigenpairs_against_64_bits(n, batch, dt):
    """Chunks of 16 steps of the inverse iteration, and groups of eight steps of
    the complex128 count.  Eigenvalues as backward stability gives them,
    (2 n + 24) u ||H||; vectors orthonormal to n u after the polish and residuals of
    the reduction's (8 n + 64) u ||H||."""
    g = torch.Generator().manual_seed(n)
    X = torch.randn(batch, n + 2, n, generator=g, dtype=torch.complex128)
    H = (X.mH @ X).to(dt)
    w, v = (t.cpu().to(torch.complex128) for t in ops.heevd(H.to(DEV)))
    u = 2.0 ** -24 if dt == torch.complex64 else 2.0 ** -53
    for b in range(batch):
        A = H[b].to(torch.complex128)
        ref = torch.linalg.eigvalsh(A).flip(0)
        top = float(ref.abs().max())
        assert float((w[b].real - ref).abs().max()) <= (2 * n + 24) * u * top
        eye = torch.eye(n, dtype=torch.complex128)
        assert float((v[b].mH @ v[b] - eye).abs().max()) <= (2 * n + 24) * u
        assert float(torch.linalg.vector_norm(A @ v[b] - v[b] * w[b], dim=0).max()) <= (8 * n + 64) * u * top


@pytest.mark.parametrize("dt", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("chiL,chiM,chiR", [(1, 2, 2), (15, 4, 40), (16, 9, 33), (33, 70, 33), (100, 8, 3), (257, 5, 64)])
def test_split_norms(chiL, chiM, chiR, dt):
    g = torch.Generator().manual_seed(chiL + chiR)
    A = torch.randn(chiL, 2, chiM, generator=g, dtype=torch.complex128).to(dt)
    B = torch.randn(chiM, 2, chiR, generator=g, dtype=torch.complex128).to(dt)
    U = torch.linalg.qr(torch.randn(4, 4, generator=g, dtype=torch.complex128))[0].to(dt)
    m = AdaptiveMPS(2, bond_dim=1, eps_bond=0.0, chi_max_per_bond=1024, device=DEV, dtype=dt)
    m._tensors = [A.to(DEV), B.to(DEV)]
    # the one-kernel form of small gates sums by itself: a gate above its sizes shares the batch
    big = AdaptiveMPS(2, bond_dim=1, eps_bond=0.0, chi_max_per_bond=1024, device=DEV, dtype=dt)
    big._tensors = [torch.randn(40, 2, 3, generator=g, dtype=torch.complex128).to(DEV, dt),
                    torch.randn(3, 2, 40, generator=g, dtype=torch.complex128).to(DEV, dt)]
    r = amod._run_pipeline([(m, 0, U.to(DEV)), (big, 0, U.to(DEV))], dt, None, spectra=True)[0]
    f = torch.complex128
    X = torch.einsum("PQpq,apm,mqb->aPQb", U.to(f).reshape(2, 2, 2, 2), A.to(f), B.to(f))
    size = torch.einsum("PQpq,apm,mqb->aPQb", U.abs().to(f).reshape(2, 2, 2, 2), A.abs().to(f), B.abs().to(f)).real
    u = 2.0 ** -24 if dt == torch.complex64 else 2.0 ** -53
    err = (chiM + 4) * u * 2 * float((X.abs() * size).sum())
    total = float((X.abs() ** 2).sum())
    n = 2 * chiR
    assert abs(r["total"] - total) <= err
    kept = float(np.sum(r["sigma"] ** 2))
    assert abs(kept - total) <= err + (2 * n + 24) * u * total

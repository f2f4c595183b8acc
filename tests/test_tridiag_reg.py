"""The register-resident tridiagonalisation (csrc/tridiag_reg.cu) at the edges of
its forms: row groups and CTAs per matrix change at n = 32, 64, 128, 256 and
512, the last column pair is half empty at odd n, and a forced cluster size
moves rows from registers to shared memory and to L2.

The eigenvalues (tridiagonalisation, then bisection) are compared with
LAPACK's in 64 bits.  Tolerance: Householder tridiagonalisation is backward
stable, |dlambda| <= c n u ||H|| with a small constant; with c = 2 and bisection's
own 2 eps + 4 eps of the Gershgorin interval, (2 n + 24) u ||H||, u = 2^-24."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from atlasq_gb300 import _lib, ops  # noqa: E402

DEV = "cuda:0"
FORMS = [(n, 0) for n in (1, 2, 3, 31, 32, 33, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 700)] + \
        [(129, 1), (200, 2), (257, 3), (300, 1), (300, 5), (384, 16), (513, 8), (1022, 16)]


@pytest.mark.parametrize("n,C", FORMS)
def test_eigenvalues_against_64_bits(n, C):
    g = torch.Generator().manual_seed(n + 1000 * C)
    X = torch.complex(torch.randn(2, n + 2, n, generator=g, dtype=torch.float64),
                      torch.randn(2, n + 2, n, generator=g, dtype=torch.float64))
    H = X.mH @ X
    H[1] = torch.diag_embed(torch.arange(1, n + 1).to(torch.complex128))  # every column already reduced
    lib = _lib.load()
    if C:
        rc = lib.agb_set_tridiag_cluster(_lib.AGB_C64, n, 2, C, 512)
        if rc == _lib.AGB_ERR_UNSUPPORTED:
            pytest.skip("the device does not schedule this cluster size")
        assert rc == 0
    try:
        w, _ = ops.heevd(H.to(torch.complex64).to(DEV))
        w = w.cpu().double().numpy()
    finally:
        if C:
            assert lib.agb_set_tridiag_cluster(_lib.AGB_C64, n, 2, 0, 512) == 0
    for b in range(2):
        ref = np.linalg.eigvalsh(H[b].to(torch.complex64).to(torch.complex128).numpy())[::-1]
        assert np.max(np.abs(w[b] - ref)) <= (2 * n + 24) * 2.0 ** -24 * np.abs(ref).max()

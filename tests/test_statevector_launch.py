"""The one-launch dense read-out (csrc/statevec.cu) against the product per site.

Both sum over each bond in order with the same multiply-adds, so the amplitudes
have to be equal bit for bit.  The chains lie where the launch can go wrong: two
sites, odd and ragged bonds, bonds wider than the ends allow, rows that fill the
buffer, and chains on either side of the rule."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from atlasq_gb300 import ops  # noqa: E402

DEV = "cuda:0"


def _full(n, top):
    return [min(2 ** min(s, n - s), top) for s in range(n + 1)]


CHAINS = [([1, 1, 1], True), ([1, 7, 1], True), ([1, 2, 3, 2, 1], True), (_full(6, 64), True),
          (_full(10, 64), True), ([1, 5, 33, 17, 64, 3, 9, 2, 1], True), (_full(14, 128), True),
          ([1, 700, 700, 1], True), (_full(20, 2), True), (_full(20, 4), True), (_full(20, 64), False),
          ([1, 3000, 3000, 1], False)]


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("chi,fits", CHAINS)
def test_amplitudes_equal_the_products(chi, fits, dtype):
    g = torch.Generator().manual_seed(sum(chi))
    T = [torch.randn(chi[s], 2, chi[s + 1], generator=g, dtype=torch.complex128).to(DEV, dtype)
         for s in range(len(chi) - 1)]
    psi = ops.statevector(T)
    assert (psi is not None) == fits
    if fits:
        ref = T[0].reshape(2, -1)
        for t in T[1:]:
            ref = ops.cgemm(ref.contiguous(), t.reshape(t.shape[0], -1)).reshape(-1, t.shape[2])
        assert torch.equal(psi, ref.reshape(-1))

"""Two factorisations in one launch (agb_qr_pair), and the canonical form that pairs
the sweeps from both ends: bit for bit the results of one after the other, where the
two take one launch (equal cluster sizes, equal and unequal row counts) and where
they do not (small matrices, unequal cluster sizes)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from atlasq_gb300 import AdaptiveMPS, ops  # noqa: E402

DEV = "cuda:0"


def _rnd(g, dt, *shape):
    return torch.randn(*shape, generator=g, dtype=torch.complex128).to(DEV, dt)


@pytest.mark.parametrize("dt", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("a,b", [((512, 256), (512, 256)), ((120, 250), (600, 250)), ((257, 100), (130, 100)),
                                 ((512, 256), (64, 64)), ((4, 2), (512, 256)), ((4, 2), (2, 2))])
def test_pair_equals_singles(a, b, dt):
    g = torch.Generator().manual_seed(a[0] + b[1])
    A, B = _rnd(g, dt, *a), _rnd(g, dt, b[1], b[0])
    (Q, R), (Q2, R2) = ops.qr_pair(A, B)
    S, S2 = ops.qr(A), ops.qr(B, transA=True, trans_out=True)
    for x, y in ((Q, S[0]), (R, S[1]), (Q2, S2[0]), (R2, S2[1])):
        assert torch.equal(x, y)


@pytest.mark.parametrize("center", [0, 1, 3, 5, 6])
def test_mixed_form_equals_sequential(center):
    n, chi = 7, [1, 2, 70, 100, 33, 64, 2, 1]
    g = torch.Generator().manual_seed(center)
    T = [_rnd(g, torch.complex64, chi[s], 2, chi[s + 1]) for s in range(n)]
    m = AdaptiveMPS(n, bond_dim=1, chi_max_per_bond=128, device=DEV)
    m.tensors, m.bond_dims = [t.clone() for t in T], chi[1:-1]
    m.to_mixed_canonical(center)
    for i in range(center):
        Q, R = ops.qr(T[i].reshape(-1, T[i].shape[2]))
        T[i] = Q.reshape(T[i].shape[0], 2, -1)
        T[i + 1] = ops.cgemm(R, T[i + 1].reshape(T[i + 1].shape[0], -1)).reshape(R.shape[0], 2, -1)
    for j in range(n - 1, center, -1):
        Q, R = ops.qr(T[j].reshape(T[j].shape[0], -1), transA=True, trans_out=True)
        T[j] = Q.reshape(Q.shape[0], 2, -1)
        T[j - 1] = ops.cgemm(T[j - 1].reshape(-1, T[j - 1].shape[2]), R).reshape(T[j - 1].shape[0], 2, -1)
    assert all(torch.equal(a, b) for a, b in zip(m.tensors, T))
    assert m.bond_dims == [t.shape[2] for t in T[:-1]]

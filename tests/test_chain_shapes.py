"""Expectation values pass pointers and bonds to the kernels: chains whose bonds
disagree, and operators off the chain, are refused before any pointer is taken
(and so on host tensors too, which no kernel could read)."""
import types

import pytest
import torch

from atlasq_gb300.mpo_ops import MPO, environments, expectation_value, local_expectations

Z = torch.tensor([[1, 0], [0, -1]], dtype=torch.complex64)


def _mps(*shapes, device="cpu"):
    return types.SimpleNamespace(num_qubits=len(shapes),
                                 tensors=[torch.ones(s, dtype=torch.complex64, device=device) for s in shapes])


CHAINS = {
    "bonds": ((1, 2, 8), (4, 2, 2), (2, 2, 1)),       # site 0 wider than site 1
    "bonds_up": ((1, 2, 2), (4, 2, 2), (2, 2, 1)),
    "left_boundary": ((2, 2, 2), (2, 2, 1)),
    "physical": ((1, 3, 2), (2, 2, 1)),
    "no_matrix": ((1, 2), (2, 2, 1)),
}


@pytest.mark.parametrize("shapes", CHAINS.values(), ids=CHAINS)
def test_disagreeing_chains_are_refused(shapes):
    m = _mps(*shapes)
    for call in (lambda: environments(m), lambda: local_expectations(m, [{0: Z}]),
                 lambda: expectation_value(MPO.identity(len(shapes), device="cpu"), m)):
        with pytest.raises(ValueError, match="site"):
            call()


def test_open_right_boundary_is_refused_by_environments():
    m = _mps((1, 2, 2), (2, 2, 3))
    for call in (lambda: environments(m), lambda: local_expectations(m, [{0: Z}])):
        with pytest.raises(ValueError, match="right boundary"):
            call()


def test_operator_bonds_that_do_not_meet_are_refused():
    mpo = MPO.identity(3, device="cpu")
    mpo.tensors[0] = torch.ones(1, 2, 2, 3, dtype=torch.complex64)  # three channels leave, one arrives
    with pytest.raises(ValueError, match="MPO site 1"):
        expectation_value(mpo, _mps((1, 2, 2), (2, 2, 2), (2, 2, 1)))


def test_host_tensors_and_missing_sites_are_refused():
    m = _mps((1, 2, 2), (2, 2, 1))
    with pytest.raises(ValueError, match="CUDA"):
        environments(m)
    m.num_qubits = 3
    with pytest.raises(IndexError):
        expectation_value(MPO.identity(3, device="cpu"), m)


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")
def test_observables_off_the_chain_are_refused():
    m = _mps((1, 2, 2), (2, 2, 1), device="cuda:0")
    for sites in ((-1,), (2,), (0, 2)):
        with pytest.raises(IndexError):
            local_expectations(m, [{s: Z for s in sites}])
    with pytest.raises(RuntimeError):
        local_expectations(m, [{0: Z[:1, :1]}])


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")
def test_open_ends_that_were_taken_stay_taken():
    """A wider first operator tensor counts by its leading channel, an open right
    boundary by its first entry: 64-bit einsums of that rule.  Bound: a chain of n
    sites of sums of 4 chi + 8 terms, as in test_expectation_lists.py."""
    g = torch.Generator().manual_seed(3)
    shapes = ((1, 2, 3), (3, 2, 4), (4, 2, 2))
    m = _mps(*shapes, device="cuda:0")
    m.tensors = [torch.complex(torch.randn(s, generator=g), torch.randn(s, generator=g)).to("cuda:0") for s in shapes]
    mpo = MPO.identity(3, device="cuda:0")
    mpo.tensors = [torch.complex(torch.randn(s, generator=g), torch.randn(s, generator=g)).to("cuda:0")
                   for s in ((2, 2, 2, 3), (4, 2, 2, 2), (2, 2, 2, 2))]
    E = torch.ones(1, 1, 1, dtype=torch.complex128, device="cuda:0")
    N, size = E[0], E.real
    for A, W in zip((t.to(torch.complex128) for t in m.tensors), (t.to(torch.complex128) for t in mpo.tensors)):
        W = W[:E.shape[0]]
        E = torch.einsum("Lab,atr,LstR,bsB->RrB", E, A.conj(), W, A)
        size = torch.einsum("Lab,atr,LstR,bsB->RrB", size, A.abs(), W.abs(), A.abs())
        N = torch.einsum("ab,asr,bsB->rB", N, A.conj(), A)
    got, want = expectation_value(mpo, m), complex(E[0, 0, 0] / N[0, 0])
    assert abs(got - want) <= 2 * 3 * (4 * 4 + 8) * 2.0 ** -24 * float(size[0, 0, 0] / N[0, 0].abs())

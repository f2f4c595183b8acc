"""Observables in launch lists: supports of every length (gaps included), uneven
bonds on both sides of the tensor-core limit of 32, operators on the host and on
the device, more observables than one list holds, and an MPO of uneven bonds,
against 64-bit einsums over the same tensors.

Tolerance: an environment chain of n sites in working precision u is within
n (4 chi + 8) u of the sum of magnitudes; values are divided by the norm, so the
bound is 2 n (4 chi + 8) u relative to the operators' norm product, with the
tensor cores' accumulation (2e-9 K per product) added for complex64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import atlasq_gb300 as aq  # noqa: E402

DEV = "cuda:0"


def _state(dims, dt, seed):
    g = torch.Generator().manual_seed(seed)
    d = [1] + list(dims) + [1]
    T = [torch.complex(torch.randn(d[i], 2, d[i + 1], generator=g, dtype=torch.float64),
                       torch.randn(d[i], 2, d[i + 1], generator=g, dtype=torch.float64)) / np.sqrt(4 * d[i + 1])
         for i in range(len(d) - 1)]
    m = aq.AdaptiveMPS(len(T), bond_dim=1, device=DEV, dtype=dt, dtype_policy=aq.DTypePolicy(default=dt))
    m.tensors = [t.to(dt).to(DEV) for t in T]
    m.bond_dims = list(dims)
    return m, [t.to(dt).to(torch.complex128) for t in T]


def _value(T, ops):
    """<psi| prod O^T |psi> / <psi|psi>: the ket is contracted on an operator's first index."""
    def sweep(W):
        E = torch.ones(1, 1, dtype=torch.complex128)
        for i, A in enumerate(T):
            E = torch.einsum("ab,atr,st,bsB->rB", E, A.conj(), W.get(i, torch.eye(2, dtype=torch.complex128)), A)
        return E[0, 0]
    return complex(sweep(ops) / sweep({}))


def _tol(dims, dt):
    u = 2.0 ** -24 if dt == torch.complex64 else 2.0 ** -53
    n, chi = len(dims) + 1, max(dims)
    return 2 * n * ((4 * chi + 8) * u + (4e-9 * chi if dt == torch.complex64 else 0))


@pytest.mark.parametrize("dt", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("dims,count", [((2, 3, 5, 7, 4, 2), 40), ((2, 4, 31, 33, 40, 17, 2), 12), ((2, 2), 600)])
def test_local_expectations_against_64_bits(dims, count, dt):
    m, T = _state(dims, dt, len(dims))
    n = len(T)
    g = torch.Generator().manual_seed(count)
    obs, want = [], []
    for k in range(count):
        a, b = sorted(torch.randint(0, n, (2,), generator=g).tolist())
        sites = {a, b} if k % 3 else set(range(a, b + 1))
        o = {}
        for i in sites:
            q = torch.linalg.qr(torch.complex(torch.randn(2, 2, generator=g, dtype=torch.float64),
                                              torch.randn(2, 2, generator=g, dtype=torch.float64)))[0].to(dt)
            o[i] = q.to(DEV) if k % 5 == 1 else q
        obs.append(o)
        want.append(o)
    got = np.array(aq.local_expectations(m, obs))
    pick = range(count) if count <= 40 else (0, 1, 511, 512, 599)
    for k in pick:
        ref = _value(T, {i: q.cpu().to(torch.complex128) for i, q in want[k].items()})
        assert abs(got[k] - ref) <= _tol(dims, dt), (k, got[k], ref)


@pytest.mark.parametrize("dt", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("dims,wdims", [((2, 3, 5), (1, 4, 2)), ((2, 4, 33, 40, 2), (3, 1, 5, 2, 1))])
def test_mpo_expectation_against_64_bits(dims, wdims, dt):
    m, T = _state(dims, dt, 9)
    g = torch.Generator().manual_seed(3)
    w = [1] + list(wdims) + [1]
    W = [torch.complex(torch.randn(w[i], 2, 2, w[i + 1], generator=g, dtype=torch.float64),
                       torch.randn(w[i], 2, 2, w[i + 1], generator=g, dtype=torch.float64)).to(dt) for i in range(len(T))]
    got = aq.expectation_value(aq.MPO(W), m)  # host tensors: converted as before
    E = torch.ones(1, 1, 1, dtype=torch.complex128)
    mag = torch.ones(1, 1, 1, dtype=torch.float64)
    N = torch.ones(1, 1, dtype=torch.complex128)
    for A, w_ in zip(T, W):
        w64 = w_.to(torch.complex128)
        E = torch.einsum("Lab,atr,LstR,bsB->RrB", E, A.conj(), w64, A)
        mag = torch.einsum("Lab,atr,LstR,bsB->RrB", mag, A.abs(), w64.abs(), A.abs())
        N = torch.einsum("ab,asr,bsB->rB", N, A.conj(), A)
    scale = float(mag.reshape(-1)[0] / N.abs().reshape(-1)[0])
    assert abs(got - complex(E.reshape(-1)[0] / N.reshape(-1)[0])) <= _tol(dims, dt) * scale

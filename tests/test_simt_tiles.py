"""Tile edges of the SIMT kernels that choose a tile by type or size: the gate
contraction (8 x 8 tiles for complex128, 16 x 16 and, for large grids, 32 x 32 for
complex64), the complex128 GEMM (16 x 16, K-step 16) and the complex64 one (64 x
64 for large grids, else 32 x 32).  Against 64-bit (or
wider than 64-bit for complex128: componentwise bound) references: a sum of K
products in the working precision is within 2 K u of the sum of magnitudes
(two multiply-adds per real product pair), plus 8 u for the 4 x 4 gate."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from atlasq_gb300 import ops  # noqa: E402

DEV = "cuda:0"


def _c(shape, gen):
    return torch.complex(torch.randn(shape, generator=gen, dtype=torch.float64),
                         torch.randn(shape, generator=gen, dtype=torch.float64))


@pytest.mark.parametrize("L,M,R", [(1, 1, 1), (7, 15, 9), (8, 16, 8), (17, 33, 31), (577, 17, 576), (600, 3, 513)])
@pytest.mark.parametrize("dt", [torch.complex64, torch.complex128])
def test_contract_gate_tiles(L, M, R, dt):
    g = torch.Generator().manual_seed(L + M + R)
    A, B, U = _c((L, 2, M), g).to(dt), _c((M, 2, R), g).to(dt), _c((4, 4), g).to(dt)
    got = ops.contract_gate(A.to(DEV), B.to(DEV), U.to(DEV)).cpu().to(torch.complex128).reshape(L, 2, 2, R)
    a, b, u = (t.to(torch.complex128) for t in (A, B, U))
    th = torch.einsum("apm,mqb->apqb", a, b)
    ref = torch.einsum("PQpq,apqb->aPQb", u.reshape(2, 2, 2, 2), th)
    mag = torch.einsum("PQpq,apqb->aPQb", u.abs().reshape(2, 2, 2, 2), torch.einsum("apm,mqb->apqb", a.abs(), b.abs()))
    unit = 2.0 ** -24 if dt == torch.complex64 else 2.0 ** -53
    # the complex128 reference has the same rounding as the result: twice the bound
    assert bool(((got - ref).abs() <= 2 * (2 * M + 8) * unit * mag).all())


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (15, 17, 16), (16, 16, 15), (33, 31, 47), (70, 96, 96), (65, 9700, 17),
                                   (20000, 33, 31)])
@pytest.mark.parametrize("opA,opB", [("N", "N"), ("C", "T"), ("R", "C")])
@pytest.mark.parametrize("dt", [torch.complex64, torch.complex128])
def test_gemm_tiles(M, N, K, opA, opB, dt):
    g = torch.Generator().manual_seed(M + N + K)
    A, B = _c((M, K) if opA in "NR" else (K, M), g).to(dt), _c((K, N) if opB in "NR" else (N, K), g).to(dt)
    f = {"N": lambda x: x, "T": lambda x: x.T, "C": lambda x: x.mH, "R": lambda x: x.conj()}
    got = ops.cgemm(A.to(DEV), B.to(DEV), opA, opB).cpu().to(torch.complex128)
    a, b = f[opA](A.to(torch.complex128)), f[opB](B.to(torch.complex128))
    unit = 2.0 ** -24 if dt == torch.complex64 else 2.0 ** -53
    assert bool(((got - a @ b).abs() <= 2 * 2 * K * unit * (a.abs() @ b.abs())).all())

"""The tensor-core GEMM's operand reads and its epilogue at the layouts where they
branch: bases and row strides that are not 16-byte aligned (scalar instead of
vector reads), partial last slices, ragged tile edges, and C = alpha AB + beta C.
Tolerance as for the other tensor-core GEMM tests: 1e-6 + 2e-9 K (the fp32
accumulation error grows with K)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from atlasq_gb300 import ops  # noqa: E402

DEV = "cuda:0"


def _at(shape, shift, gen):
    """A contiguous tensor that starts `shift` complex numbers into its storage."""
    n = int(np.prod(shape))
    buf = torch.complex(torch.randn(n + shift, generator=gen), torch.randn(n + shift, generator=gen)).to(DEV)
    return buf[shift:].view(*shape)


@pytest.mark.parametrize("opA,opB", [("N", "N"), ("C", "N"), ("N", "T"), ("C", "R")])
@pytest.mark.parametrize("M,N,K", [(128, 64, 64), (129, 65, 65), (31, 33, 32), (257, 190, 100)])
@pytest.mark.parametrize("sa,sb", [(0, 0), (1, 0), (0, 1)])
def test_layouts(opA, opB, M, N, K, sa, sb):
    g = torch.Generator().manual_seed(M * N + K)
    A = _at((M, K) if opA in "NR" else (K, M), sa, g)
    B = _at((K, N) if opB in "NR" else (N, K), sb, g)
    C = _at((M, N), 1, g)
    a, b = A.cpu().to(torch.complex128), B.cpu().to(torch.complex128)
    f = {"N": lambda x: x, "T": lambda x: x.T, "C": lambda x: x.mH, "R": lambda x: x.conj()}
    prod = f[opA](a) @ f[opB](b)
    ref = (0.5 - 0.25j) * prod + (1.5 + 0.5j) * C.cpu().to(torch.complex128)
    tol = 1e-6 + 2e-9 * K
    got = ops.cgemm_tc(A, B, opA, opB).cpu().to(torch.complex128)
    assert torch.linalg.norm(got - prod) <= tol * torch.linalg.norm(prod)
    got = ops.cgemm_tc(A, B, opA, opB, alpha=0.5 - 0.25j, beta=1.5 + 0.5j, C=C).cpu().to(torch.complex128)
    assert torch.linalg.norm(got - ref) <= tol * torch.linalg.norm(ref)

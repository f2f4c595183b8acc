"""The shared-memory form of the small QR (csrc/qr.cu, M N < 64 x 64) against the
global-memory kernel that agb_qr_noalloc runs: the same sums in the same order, so
Q and R have to be equal bit for bit.  Single rows and columns, sizes around the
groups of four columns and eight rows, the largest of the range, a zero column and a
matrix that is triangular already."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from atlasq_gb300 import _lib, ops  # noqa: E402

DEV = "cuda:0"
SHAPES = [(1, 1), (1, 7), (7, 1), (2, 2), (4, 4), (5, 3), (8, 9), (9, 8), (16, 16), (17, 33), (33, 17), (64, 32), (63, 65),
          (65, 63), (31, 132), (132, 31), (4095, 1), (1, 4095), (2, 2047), (2047, 2), (1100, 3)]


@pytest.mark.parametrize("dt", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("M,N", SHAPES)
def test_equals_the_global_memory_kernel(M, N, dt, trans):
    g = torch.Generator().manual_seed(M + 7 * N)
    A = torch.randn(M, N, generator=g, dtype=torch.complex128)
    mats = [A, torch.triu(A)]
    zero = A.clone()
    zero[:, N // 2] = 0
    mats.append(zero)
    lib = _lib.load()
    k = min(M, N)
    for a in mats:
        a = (a.T.contiguous() if trans else a).to(DEV, dt)
        Q, R = ops.qr(a, transA=trans, trans_out=trans)
        Qn, Rn = torch.empty_like(Q), torch.empty_like(R)
        assert Q.shape == ((k, M) if trans else (M, k))
        _lib.check(lib.agb_qr_noalloc(_lib.dtype_code(dt), _lib.ptr(a), M, N, int(trans), _lib.ptr(Qn), _lib.ptr(Rn),
                                      int(trans), _lib.stream_ptr(torch.device(DEV))), "qr_noalloc")
        assert torch.equal(Q, Qn)
        assert torch.equal(R, Rn)

"""Both sides of the product list's choice of kernel: groups whose 32 x 32 tiles find
an SM each (SIMT GEMM) and larger ones (tcgen05), mixed with small and ragged
products, over all operand forms.  A sum of K products in float32 is within 2 K u
of the sum of magnitudes; the 3xTF32 split drops products below 2^-21 of each term
and truncates its sums: 64 u more (u = 2^-24)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from atlasq_gb300 import ops  # noqa: E402

DEV = torch.device("cuda:0")
FORM = {"N": lambda t: t, "T": lambda t: t.mT, "C": lambda t: t.mH, "R": lambda t: t.conj()}


@pytest.mark.parametrize("dt", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("shapes", [[(32, 32, 32)], [(33, 65, 31), (1, 1, 1)], [(256, 608, 40)], [(256, 609, 40)],
                                    [(130, 257, 100), (64, 64, 300), (5, 200, 7)], [(300, 300, 64), (300, 200, 96), (2, 2, 2)]])
def test_both_sides(shapes, dt):
    g = torch.Generator().manual_seed(len(shapes) + shapes[0][1])
    forms = [(a, b) for a in "NTCR" for b in "NTC"] if len(shapes) == 1 and shapes[0][1] < 100 else [("N", "N"), ("C", "N"), ("N", "C")]
    for fa, fb in forms:
        prods, keep = [], []
        for M, N, K in shapes:
            A = torch.randn(*((M, K) if fa in "NR" else (K, M)), generator=g, dtype=torch.complex128).to(dt)
            B = torch.randn(*((K, N) if fb in "NR" else (N, K)), generator=g, dtype=torch.complex128).to(dt)
            a, b = A.to(DEV), B.to(DEV)
            d = torch.empty(M, N, dtype=dt, device=DEV)
            keep.append((A, B, a, b, d))
            prods.append((M, N, K, fa, fb, a.data_ptr(), a.shape[1], b.data_ptr(), b.shape[1], d.data_ptr(), N))
        lst = ops.ProductList(dt, DEV)
        n = lst.group(prods)
        lst.upload().launch(n)
        u = 2.0 ** -24 if dt == torch.complex64 else 2.0 ** -53
        for (M, N, K), (A, B, _, _, d) in zip(shapes, keep):
            A, B = FORM[fa](A.to(torch.complex128)), FORM[fb](B.to(torch.complex128))
            ref, mag = A @ B, A.abs() @ B.abs()
            # complex128: the reference rounds like the result
            assert bool(((d.cpu().to(torch.complex128) - ref).abs() <= 2 * (2 * K + 64) * u * mag).all())

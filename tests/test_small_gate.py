"""The one-kernel vector phase of small complex64 gates (csrc/small_gate.cuh: m, n,
ell <= 64) against the batched kernels, which the same gates take when a larger
gate shares their batch.

Tolerances (u = 2^-24, X the gate's matrix, K = max(m, n, chiM)).  sigma^2: the
contraction rounds X by (chiM + 4) u, the reduction and bisection add 2 n + 24, so
each side is within (2 n + 2 chiM + 32) u ||X||^2 of the true value.  Product of
the split without truncation: the basis is orthonormal to n u after the polish
and each contraction and the application of the gate rounds K u, so
||A' B' - X|| <= (4 K + 24) u ||X||; with truncation the weight left out is the
true tail to within the sigma^2 tolerance."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from atlasq_gb300 import AdaptiveMPS, _lib  # noqa: E402
from atlasq_gb300 import adaptive_mps as amod  # noqa: E402

DEV = "cuda:0"
C64, C128 = torch.complex64, torch.complex128


def _entry(chiL, chiM, chiR, cap, eps, decay, seed):
    """A two-site chain whose pair has the given bonds; ``decay`` shapes its spectrum."""
    g = torch.Generator().manual_seed(seed)
    rnd = lambda *s: torch.complex(torch.randn(*s, generator=g, dtype=torch.float64),  # noqa: E731
                                   torch.randn(*s, generator=g, dtype=torch.float64))
    m = AdaptiveMPS(2, bond_dim=1, eps_bond=eps, chi_max_per_bond=cap, device=DEV, dtype=C64)
    scale = decay ** torch.arange(chiM, dtype=torch.float64)
    A = (rnd(chiL, 2, chiM) * scale).to(C64)
    B = rnd(chiM, 2, chiR).to(C64)
    U = torch.linalg.qr(rnd(4, 4))[0].to(C64)
    X = torch.einsum("PQpq,apm,mqb->aPQb", U.to(C128).reshape(2, 2, 2, 2), A.to(C128),
                     B.to(C128)).reshape(2 * chiL, 2 * chiR).numpy()
    m._tensors = [A.to(DEV), B.to(DEV)]
    return (m, 0, U.to(DEV)), X


SHAPES = [(1, 1, 1), (1, 2, 2), (2, 3, 1), (3, 5, 7), (8, 16, 8), (16, 16, 17), (31, 8, 32), (32, 32, 32), (32, 4, 5)]


def _run(cases, extra):
    entries, Xs = zip(*[_entry(*c) for c in cases])
    entries = list(entries) + ([_entry(33, 4, 33, 64, 1e-6, 1.0, 99)[0]] if extra else [])
    return amod._run_pipeline(entries, C64, None, spectra=True)[:len(cases)], entries, Xs


@pytest.mark.parametrize("cap,eps,decay", [(64, 0.0, 1.0), (64, 1e-3, 0.6), (4, 1e-6, 0.8), (64, 1e-2, 0.3)])
def test_one_kernel_against_batched(cap, eps, decay):
    cases = [(*s, cap, eps, decay, 7 * i + 1) for i, s in enumerate(SHAPES)]
    small, entries, Xs = _run(cases, False)
    batched, _, _ = _run(cases, True)
    for r, q, (m, _, _), X in zip(small, batched, entries, Xs):
        n, u = X.shape[1], 2.0 ** -24
        chiM = m.tensors[0].shape[2]
        K, norm2 = max(*X.shape, chiM), np.linalg.norm(X) ** 2
        tol = (2 * n + 2 * chiM + 32) * u * norm2
        assert (r["status"], r["ell"]) == (q["status"], q["ell"]) == (_lib.AGB_OK, min(cap, *X.shape))
        ref = np.linalg.svd(X, compute_uv=False) ** 2
        c = min(len(r["sigma"]), len(q["sigma"]), len(ref))
        assert np.max(np.abs(r["sigma"][:c] ** 2 - ref[:c])) <= tol
        assert np.max(np.abs(r["sigma"][:c] ** 2 - q["sigma"][:c] ** 2)) <= 2 * tol
        # the ranks differ at most where the weight between them is within the rounding
        lo, hi = sorted((r["k"], q["k"]))
        assert 1 <= lo and hi <= min(cap, *X.shape) and ref[lo:hi].sum() <= 2 * tol
        P = torch.einsum("apk,kqb->apqb", r["A"].cpu().to(C128), r["B"].cpu().to(C128)).reshape(X.shape).numpy()
        err2 = np.linalg.norm(P - X) ** 2
        if r["k"] == min(X.shape):
            assert err2 <= ((4 * K + 24) * u) ** 2 * norm2
        else:
            assert err2 <= ref[r["k"]:].sum() + tol

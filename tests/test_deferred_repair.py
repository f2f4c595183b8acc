"""The repair pass of the host-synchronised updates: gates too large for the one-kernel
form report that they want one, and the second call does what the call that repairs at
once does; where the first call has nothing left to do, no second one is issued.

The overlap is planted as in test_gpu_parity.py: four leading eigenvalues 2e-7
apart, solved one by one (cluster tolerance ~0)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import atlasq_gb300 as aq  # noqa: E402
from atlasq_gb300 import _lib  # noqa: E402
from atlasq_gb300 import adaptive_mps as amod  # noqa: E402

DEV = "cuda:0"


def _planted(lam, seed):
    """X = W_L diag(sqrt(lam)) W_R^H as two site tensors (identity gate)."""
    rng, nn = np.random.default_rng(seed), len(lam)

    def haar():
        q, r = np.linalg.qr(rng.standard_normal((nn, nn)) + 1j * rng.standard_normal((nn, nn)))
        return q * (np.diag(r) / np.abs(np.diag(r)))[None, :]
    A = (haar() * np.sqrt(lam)[None, :]).reshape(nn // 2, 2, nn).astype(np.complex64)
    return A, haar().conj().T.reshape(nn, 2, nn // 2).astype(np.complex64)


def _run(A, B, cap, oc, **kw):
    m = aq.AdaptiveMPS(2, bond_dim=1, eps_bond=1e-8, chi_max_per_bond=cap, device=DEV)
    m._operation_counter = oc
    m._tensors = [torch.tensor(A).to(DEV), torch.tensor(B).to(DEV)]
    m._bond_dims = [A.shape[2]]
    lib = _lib.load()
    n0 = lib.agb_launch_count()
    r = amod._run_pipeline([(m, 0, torch.eye(4, dtype=torch.complex64, device=DEV))], torch.complex64, kw.pop("ells", None),
                           **kw)[0]
    return r, lib.agb_launch_count() - n0


def _errors(A, B, r):
    X = np.einsum("apm,mqb->apqb", A.astype(np.complex128), B.astype(np.complex128)).reshape(2 * A.shape[0], -1)
    rec = np.einsum("apk,kqb->apqb", r["A"].cpu().numpy().astype(np.complex128),
                    r["B"].cpu().numpy().astype(np.complex128)).reshape(X.shape)
    s2 = np.linalg.svd(X, compute_uv=False) ** 2
    return np.linalg.norm(X - rec) / np.sqrt(s2.sum()), np.sqrt(s2[r["k"]:].sum() / s2.sum())


@pytest.mark.parametrize("half", [40, 64])
def test_second_call_repairs(half, monkeypatch):
    lam = np.concatenate([1.0 - 2e-7 * np.arange(4), 0.6 * np.exp(-np.arange(2 * half - 4) / 6.0)])
    cap, kw = 24, {"all_vectors": True, "cluster_tol": 1e-30}
    A, B = _planted(lam, 5)
    repaired = 0
    for oc in range(8):
        with monkeypatch.context() as p:  # everything in the first call
            p.setattr(_lib, "AGB_RUN_REPAIR_LATER", _lib.AGB_RUN_REPAIR)
            at_once, _ = _run(A, B, cap, oc, **kw)
        r, _ = _run(A, B, cap, oc, **kw)
        repaired += bool(r["repair"] & 2)
        assert r["status"] == 0 and r["repair"] == at_once["repair"] and r["k"] == at_once["k"]
        assert torch.equal(r["A"], at_once["A"]) and torch.equal(r["B"], at_once["B"])
        err, opt = _errors(A, B, r)
        assert err <= 2 * opt + 1e-5, (oc, err, opt)
    assert repaired >= 1


@pytest.mark.parametrize("half", [8, 64])
def test_no_second_call_without_work(half):
    """A predicted number of eigenpairs below the rank (AGB_ERR_RANK) is not the
    device's to repair."""
    A, B = _planted(np.linspace(1.0, 0.5, 2 * half), 3)
    full, launches = _run(A, B, half, 0)
    short, fewer = _run(A, B, half, 0, ells=[half // 2])
    assert full["status"] == 0 and short["status"] == _lib.AGB_ERR_RANK
    assert fewer <= launches


def test_no_second_call_after_the_one_kernel_repair():
    """m = n = 64: the repair runs inside the kernel of the small gates."""
    A, B = _planted(np.concatenate([1.0 - 2e-7 * np.arange(4), 0.6 * np.exp(-np.arange(60) / 6.0)]), 5)
    runs = [_run(A, B, 24, oc, all_vectors=True, cluster_tol=1e-30) for oc in range(8)]
    assert any(r["repair"] & 2 for r, _ in runs)
    assert len({launches for _, launches in runs}) == 1

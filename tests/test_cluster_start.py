"""Distributed shared memory may be touched only once every CTA of the cluster has
started: in each kernel a cluster barrier stands before the first access to a peer's
shared memory (read from the source; a run cannot show the order it happened to have)."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "atlasq_gb300" / "csrc"
REMOTE = re.compile(r"map_shared_rank\(|\bsend\(")
BARRIER = re.compile(r"cluster\.sync\(\)|cluster_barrier\(\)")


def _kernels():
    for f in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        for body in text.split("__global__")[1:]:
            if REMOTE.search(body):
                yield f.name, re.search(r"\w+_kernel(?=\()", body).group(0), body


@pytest.mark.parametrize("name,kernel,body", [pytest.param(*k, id=f"{k[0]}-{k[1]}") for k in _kernels()])
def test_cluster_barrier_before_the_first_remote_access(name, kernel, body):
    first, barrier = REMOTE.search(body).start(), BARRIER.search(body)
    assert barrier and barrier.start() < first, f"{name}: {kernel}"


def test_the_cluster_kernels_are_found():
    assert {n for n, _, _ in _kernels()} >= {"tridiag_reg.cu", "tridiag_cluster.cu", "tridiag_2stage.cu",
                                             "qr_cluster.cu"}


@pytest.mark.gpu
def test_one_by_one_matrix_on_a_forced_cluster():
    """A cluster size set for a size class holds for n = 1 too: only the CTA that has the
    row writes the result.  Bound (2 n + 24) u of test_tridiag_reg.py (bisection ends
    within a few u of the diagonal)."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from atlasq_gb300 import _lib, ops
    lib = _lib.load()
    H = torch.arange(1.0, 65.0).to(torch.complex128).to("cuda:0").reshape(64, 1, 1)
    for dtype, code, u in ((torch.complex64, _lib.AGB_C64, 2.0 ** -24), (torch.complex128, _lib.AGB_C128, 2.0 ** -53)):
        assert lib.agb_set_tridiag_cluster(code, 24, 64, 8, 512) == 0  # the class of n <= 32, more than 32 matrices
        try:
            w, _ = ops.heevd(H.to(dtype))
        finally:
            assert lib.agb_set_tridiag_cluster(code, 24, 64, 0, 512) == 0
        ref = H.real.reshape(-1)
        assert bool(((w.reshape(-1).double() - ref).abs() <= 26 * u * ref).all())

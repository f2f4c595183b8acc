"""Lengths of a row around those the sampling step keeps in registers (64, 128, 256
elements a half, then any).  The outcome and the probability follow from the row:
u from Philox, p = |row half|^2 summed to double accuracy, so pz is within the
float32 rounding of the squares (4 u relative, u = 2^-24; complex128: 2 chi u of
its own); the new row is the chosen half, bit for bit."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from atlasq_gb300 import _lib  # noqa: E402

DEV = torch.device("cuda:0")


@pytest.mark.parametrize("dt", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("chi", [1, 31, 33, 64, 65, 127, 128, 129, 255, 256, 257, 600])
def test_row_lengths(chi, dt):
    shots = 41
    g = torch.Generator().manual_seed(chi)
    temp = torch.randn(shots, 2 * chi, generator=g, dtype=torch.complex128).to(DEV, dt)
    bits = torch.zeros(shots, dtype=torch.int64, device=DEV)
    new = torch.empty(shots, chi, dtype=dt, device=DEV)
    pz = torch.empty(shots, dtype=torch.float64, device=DEV)
    lib = _lib.load()
    _lib.check(lib.agb_sample_site(_lib.dtype_code(dt), _lib.ptr(temp), shots, chi, 3, ctypes.c_uint64(5), ctypes.c_uint64(0),
                                   _lib.ptr(bits), _lib.ptr(new), _lib.ptr(pz), _lib.stream_ptr(DEV)), "sample_site")
    halves = temp.reshape(shots, 2, chi)
    p = (halves.to(torch.complex128).abs() ** 2).sum(2) + 1e-15
    ref = p[:, 0] / p.sum(1)
    u = 2.0 ** -24 if dt == torch.complex64 else 2 * chi * 2.0 ** -53
    assert float(((pz - ref) / ref).abs().max()) <= 8 * u
    assert bool(((bits == 0) | (bits == 1)).all())
    assert torch.equal(new, halves[torch.arange(shots, device=DEV), bits])

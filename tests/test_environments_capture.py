"""The environment sweeps take no host copy under stream capture, and the captured
products are those of the eager call (tensor-core and SIMT groups), bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import types  # noqa: E402

from atlasq_gb300.mpo_ops import environments  # noqa: E402

DEV = "cuda:0"


@pytest.mark.parametrize("dt", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("dims", [(2, 5, 3), (2, 40, 200, 300, 40)])
def test_captured_environments(dims, dt):
    g = torch.Generator().manual_seed(len(dims))
    d = (1, *dims, 1)
    m = types.SimpleNamespace(tensors=[(torch.randn(a, 2, b, generator=g, dtype=dt) / (2 * b) ** 0.5).to(DEV)
                                       for a, b in zip(d, d[1:])])
    _, L, R = environments(m)  # also the first use of every kernel and scratch buffer
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _, Lg, Rg = environments(m)
    for t in m.tensors:  # the graph reads the tensors, not the values it was captured with
        t.neg_()
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(L + R, Lg + Rg))

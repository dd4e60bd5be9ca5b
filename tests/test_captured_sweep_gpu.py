"""Sweeps recorded in a CUDA graph: a replay works on what x holds then, and on nothing of the host call that
was recorded."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,dtype", [("block8", "complex64"), ("lex", "complex64"), ("lex", "complex128")])
@pytest.mark.parametrize("nrhs", [1, 3])
def test_replayed_sweep_matches_call(cuda, order, dtype, nrhs):
    """The same launches on the same values: equal to the last bit."""
    import torch
    from h3d import _lib as L
    from h3d import ops

    n, h, npml = (26, 25, 27), (25.0, 20.0, 22.0), 4
    dt = getattr(torch, dtype)
    rd = torch.float32 if dt == torch.complex64 else torch.float64
    gen = torch.Generator(device=cuda).manual_seed(2)
    N = int(np.prod(n))
    wn = torch.rand(N, dtype=rd, device=cuda, generator=gen) * 1e-4 + 1e-4
    field = lambda: torch.view_as_complex(torch.randn(nrhs, N, 2, dtype=rd, device=cuda, generator=gen))
    x, b, o = field(), field(), L.ORDER_LEX if order == "lex" else L.ORDER_BLOCK8
    sweep = lambda: ops.kacz_sweep((n, h, npml), wn, 1.5, x, b, 1, order=o)
    sweep()  # the operator's tables are made outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = sweep()
    junk = [np.full(m, 0x5A, dtype=np.uint8) for m in (64, 256, 512, 1024, 4096) for _ in range(50)]
    for _ in range(3):
        x.copy_(field())
        b.copy_(field())
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, sweep())
    del junk, graph

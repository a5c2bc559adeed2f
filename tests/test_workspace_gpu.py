"""Workspaces that grow while a captured graph still works in them (GPU)."""

import pytest
import torch

from pare_b200.decode import synthetic_linear
from pare_b200.kernels import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 8, 16, 64])
def test_graph_survives_a_larger_call_on_its_stream(rows, cuda_lib):
    """A linear is captured, then a call that needs more scratch runs on the same stream and other tensors take what memory there is:
    the replayed graph gives the same bits and leaves those tensors alone."""
    layer, x = synthetic_linear(4096, 4096, seed=3, device="cuda"), torch.randn(rows, 4096, device="cuda").half()
    tall = torch.randn(2000, 4096, device="cuda").half()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        want = layer(x)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out = layer(x)
        before = _lib.workspace(x.device, 1).numel()
        _lib.workspace(x.device, before + 1)
        layer(tall)
        others = [torch.full((before,), 255, dtype=torch.uint8, device="cuda") for _ in range(4)]
        for _ in range(3):
            out.zero_()
            graph.replay()
            assert torch.equal(out, want)
        assert all(bool((t == 255).all()) for t in others)

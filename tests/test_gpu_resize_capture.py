"""Resizing where the separable kernel does not serve (2-D images, float64,
orders above three): enqueued without waiting for the GPU, so that it can be
captured in a CUDA graph."""
import pytest
import torch

import nitorch_b200 as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,to,dtype,order", [((1, 2, 40, 33), (61, 50), torch.float32, 3),
                                                  ((1, 1, 17, 12, 20), (25, 18, 31), torch.float64, 1),
                                                  ((1, 1, 17, 12, 20), (25, 18, 31), torch.float32, 4)])
def test_capture(shape, to, dtype, order):
    x = torch.randn(shape, dtype=dtype, device="cuda")
    call = lambda: nb.resize(x, shape=to, interpolation=order, bound="dct2", dim=len(to))  # noqa: E731
    first = call()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = call()
    x.normal_()
    graph.replay()
    assert torch.equal(out, call()) and not torch.equal(out, first)

"""Bricks that hold far more samples than their share, which are cut into
chunks: grids that zoom into a few voxels, small sources, points piled outside
the volume, counts around a chunk's 1024 (scatter) and 2048 (gather) samples,
chunks that end with a brick, a batch item or the samples.  Against the FP64
oracle: gathers float32 1e-5 of max |ref|, sums of up to n = 35000 terms
sqrt(n) 2^-23 + 1e-5."""
import numpy as np
import pytest
import torch

from nitorch_b200 import _lib, spatial
from oracle import oracle as O
from tests._gpu_ops import cu, enums, np64, relerr

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _sorted():
    spatial.set_sample_order("sorted")
    yield
    spatial.set_sample_order("auto")


def _grid(kind, size, src, N, r):
    n = int(np.prod(size))
    src = np.array(src, np.float64)
    if kind == "voxel":      # every sample in one cell
        g = 0.4 * src + r.uniform(0, 0.9, (N, n, 3))
    elif kind == "zoom":     # about three voxels across, over several bricks
        g = 0.4 * src + r.uniform(-1.5, 1.5, (N, n, 3))
    elif kind == "source":   # the whole (small) source, past its edges
        g = r.uniform(-1, 1, (N, n, 3)) + r.uniform(0, 1, (N, n, 3)) * (src - 1)
    else:                    # "outside": most beyond one corner
        g = src - 1 + r.uniform(-1.5, 4, (N, n, 3))
    return g.reshape(N, *size, 3).astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("kind,size,src", [("voxel", (16, 8, 8), (9, 10, 11)), ("voxel", (32, 8, 8), (9, 10, 11)),
                                           ("voxel", (1, 31, 33), (9, 10, 11)), ("voxel", (23, 31, 33), (20, 9, 13)),
                                           ("zoom", (30, 31, 33), (20, 21, 19)), ("source", (33, 32, 32), (5, 4, 7)),
                                           ("outside", (17, 30, 33), (12, 9, 13))])
@pytest.mark.parametrize("order,C", [(3, 1), (3, 3), (2, 2), (3, 4)])
def test_dense(kind, size, src, order, C):
    r = np.random.default_rng(order + C)
    N = 2 if size[0] < 20 else 1
    grid = _grid(kind, size, src, N, r)
    vol, tgt = r.uniform(0, 1, (N, C, *src)), r.uniform(0, 1, (N, C, *size))
    b, o = enums(2, order)
    V, G, T = cu(vol, torch.float32, True), cu(grid, torch.float32, True, grid=True), cu(tgt, torch.float32, True)
    vol, tgt = np64(V), np64(T)
    args = ([2], [order], 1)
    gather, scatter = 1e-5, 1e-5 + (grid.size / 3) ** 0.5 * 2.0 ** -23

    def ran():
        assert _lib.last_kernel().startswith("pp_brick_"), _lib.last_kernel()

    assert relerr(np64(spatial.grid_pull(V, G, b, o, 1)), O.grid_pull(vol, grid, *args)) < gather
    ran()
    assert relerr(np64(spatial.grid_grad(V, G, b, o, 1)), O.grid_grad(vol, grid, *args)) < gather
    ran()
    assert relerr(np64(spatial.grid_push(T, G, list(src), b, o, 1)), O.grid_push(tgt, grid, src, *args)) < scatter
    ran()
    assert relerr(np64(spatial.grid_count(G, list(src), b, o, 1)), O.grid_count(grid, src, *args)) < scatter
    gi, gg = spatial.grid_pull_backward(T, V, G, b, o, 1)
    ran()
    ri, rg = O.grid_pull_backward(tgt, vol, grid, *args)
    assert relerr(np64(gi), ri) < scatter and relerr(np64(gg), rg) < gather
    gi, gg = spatial.grid_push_backward(V, T, G, b, o, 1)
    ran()
    ri, rg = O.grid_push_backward(vol, tgt, grid, *args)
    assert relerr(np64(gi), ri) < gather and relerr(np64(gg), rg) < gather

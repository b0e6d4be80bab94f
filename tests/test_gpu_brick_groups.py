"""The brick kernels where their grouping can go wrong, against the FP64
oracle: sources smaller than a group of 2 x 2 x 2 bricks, one voxel past a
group and many groups, quadratic and cubic stencils, every mode, samples far
outside the volume (warps full of samples that fit no window), per-sample
tensors of other layouts than the sample's index.  Tolerance: float32 1e-5
of max |ref|, bfloat16 storage 2^-8 + 1e-5."""
import numpy as np
import pytest
import torch

from nitorch_b200 import _lib, spatial
from oracle import oracle as O
from tests._cases import identity
from tests._gpu_ops import cu, enums, np64, relerr

pytestmark = pytest.mark.gpu


def _case(src, lattice, C, spread, seed, N=2):
    r = np.random.default_rng(seed)
    scale = np.array([(s - 1) / max(o - 1, 1) for s, o in zip(src, lattice)])
    grid = identity(lattice)[None] * scale + spread * r.standard_normal((N, *lattice, 3))
    grid = grid.astype(np.float32).astype(np.float64)
    return r.standard_normal((N, C, *src)), grid, r.standard_normal((N, C, *lattice))


@pytest.fixture(autouse=True)
def _sorted():
    prev = spatial._sample_order_mode
    spatial.set_sample_order("sorted")
    spatial._orders.clear()
    yield
    spatial.set_sample_order(prev)
    spatial._orders.clear()


def _check(V, G, T, bound, order, ex, tol=1e-5):
    vol, grid, tgt = np64(V), np64(G), np64(T)
    b, o, bo, oo = *enums(bound, order), [bound], [order]
    src = list(vol.shape[2:])

    def ran(name="pp_brick_"):
        k = _lib.last_kernel()
        assert k.startswith(name) and f"order={order}" in k, k

    out = spatial.grid_pull(V, G, b, o, ex)
    ran("pp_brick_gather")
    assert relerr(np64(out), O.grid_pull(vol, grid, bo, oo, ex)) < tol
    grad = spatial.grid_grad(V, G, b, o, ex)
    ran("pp_brick_gather")
    assert relerr(np64(grad), O.grid_grad(vol, grid, bo, oo, ex)) < tol
    pulled, both = spatial.grid_pull_grad(V, G, b, o, ex)
    ran("pp_brick_gather")
    assert relerr(np64(pulled), np64(out)) < 1e-6 and relerr(np64(both), np64(grad)) < 1e-6
    out = spatial.grid_push(T, G, src, b, o, ex)
    ran("pp_brick_scatter")
    assert relerr(np64(out), O.grid_push(tgt, grid, src, bo, oo, ex)) < tol
    out = spatial.grid_count(G, src, b, o, ex)
    ran("pp_brick_scatter")
    assert relerr(np64(out), O.grid_count(grid, src, bo, oo, ex)) < 1e-5
    gi, gg = spatial.grid_pull_backward(T, V, G, b, o, ex)
    ran("pp_brick_pullbwd")
    ri, rg = O.grid_pull_backward(tgt, vol, grid, bo, oo, ex)
    assert relerr(np64(gi), ri) < tol and relerr(np64(gg), rg) < 1e-5
    gi, gg = spatial.grid_push_backward(V, T, G, b, o, ex)
    ran("pp_brick_gather")
    ri, rg = O.grid_push_backward(vol, tgt, grid, bo, oo, ex)
    assert relerr(np64(gi), ri) < tol and relerr(np64(gg), rg) < 1e-5


@pytest.mark.parametrize("src", [(2, 3, 4), (8, 8, 12), (9, 17, 13), (21, 22, 27)])
@pytest.mark.parametrize("C", [1, 2, 3, 4])
@pytest.mark.parametrize("order", [2, 3])
@pytest.mark.parametrize("bound,ex,spread", [(2, 0, 1.5), (5, 1, 9.0), (3, 1, 2.0), (7, 1, 2.0)])
def test_groups(src, C, order, bound, ex, spread):
    vol, grid, tgt = _case(src, (11, 12, 14), C, spread, C + order + sum(src))
    _check(cu(vol, torch.float32, True), cu(grid, torch.float32, True), cu(tgt, torch.float32, True), bound, order, ex)


@pytest.mark.parametrize("order", [2, 3])
@pytest.mark.parametrize("C", [1, 3])
def test_bfloat16(order, C):
    vol, grid, tgt = _case((17, 16, 25), (18, 20, 23), C, 1.5, order)
    _check(cu(vol, torch.bfloat16, True), cu(grid, torch.float32, True), cu(tgt, torch.bfloat16, True), 2, order, 1,
           2.0 ** -8 + 1e-5)


def test_other_layouts():
    """Channel-last image and target, a grid whose components come first in
    memory: no tensor but the outputs is laid out by the sample's index."""
    vol, grid, tgt = _case((13, 14, 15), (9, 10, 11), 3, 2.0, 7)
    V = cu(vol, torch.float32).permute(0, 2, 3, 4, 1).contiguous().permute(0, 4, 1, 2, 3).requires_grad_()
    T = cu(tgt, torch.float32).permute(0, 2, 3, 4, 1).contiguous().permute(0, 4, 1, 2, 3).requires_grad_()
    G = cu(np.moveaxis(grid, -1, 1), torch.float32).movedim(1, -1).requires_grad_()
    _check(V, G, T, 2, 3, 1)
    T = cu(np.repeat(tgt, 2, 3), torch.float32)[:, :, :, ::2].requires_grad_()
    _check(V, G, T, 2, 3, 1)

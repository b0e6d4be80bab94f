"""The direct kernels (3-D linear and quadratic, 2-D linear to cubic, in the
grid's own order) against the FP64 oracle where their tiling can go wrong: last axes of
one voxel, shorter and longer than a tile by one, ragged middle axes, runs of
planes that end inside and across batch items, channel counts above a block,
strided and broadcast tensors.  Tolerance: float32 arithmetic 1e-5, bfloat16
storage 2^-8 + 1e-5, of max |ref| or of the inputs' scale (1) where that is
larger: gradients vanish where a bound extends the image by constants."""
import numpy as np
import pytest
import torch

from nitorch_b200 import _lib, spatial
from oracle import oracle as O
from tests._gpu_ops import cu, enums, np64

pytestmark = pytest.mark.gpu

SHAPES_3D = [(1, 1, 1), (3, 9, 1), (5, 8, 33), (2, 17, 31), (4, 5, 65)]
SHAPES_2D = [(1, 1), (9, 1), (33, 7), (8, 32), (67, 129)]


def _case(lattice, src, C, N, seed):
    r = np.random.default_rng(seed)
    dim = len(lattice)
    ident = np.stack(np.meshgrid(*[np.arange(s, dtype=np.float64) for s in lattice], indexing="ij"), -1)
    grid = ident * (np.array(src) / np.array(lattice)) + 1.2 * r.standard_normal((N, *lattice, dim))
    grid = grid.astype(np.float32).astype(np.float64)
    return r.standard_normal((N, C, *src)), grid, r.standard_normal((N, C, *lattice))


def relerr(a, ref):
    return float(np.abs(a - ref).max()) / max(1.0, float(np.abs(ref).max()))


def _check(vol, grid, tgt, bound, order, ex, dtype=torch.float32, tol=1e-5):
    b, o = enums(bound, order)
    V, G, T = cu(vol, dtype, True), cu(grid, dtype, True, grid=True), cu(tgt, dtype, True)
    vol, tgt = np64(V), np64(T)
    src = vol.shape[2:]

    def ran():
        assert _lib.last_kernel().startswith("pp_direct_kernel"), _lib.last_kernel()

    out = spatial.grid_pull(V, G, b, o, ex)
    ran()
    assert relerr(np64(out), O.grid_pull(vol, grid, [bound], [order], ex)) < tol
    out = spatial.grid_grad(V, G, b, o, ex)
    ran()
    assert relerr(np64(out), O.grid_grad(vol, grid, [bound], [order], ex)) < tol
    pulled, grad = spatial.grid_pull_grad(V, G, b, o, ex)
    assert relerr(np64(pulled), O.grid_pull(vol, grid, [bound], [order], ex)) < tol
    assert relerr(np64(grad), np64(out)) < 1e-6
    out = spatial.grid_push(T, G, list(src), b, o, ex)
    ran()
    assert relerr(np64(out), O.grid_push(tgt, grid, src, [bound], [order], ex)) < tol
    out = spatial.grid_count(G, list(src), b, o, ex)
    ran()
    assert relerr(np64(out), O.grid_count(grid, src, [bound], [order], ex)) < 1e-5
    gi, gg = spatial.grid_pull_backward(T, V, G, b, o, ex)
    ran()
    ri, rg = O.grid_pull_backward(tgt, vol, grid, [bound], [order], ex)
    assert relerr(np64(gi), ri) < tol and relerr(np64(gg), rg) < 1e-5
    gi, gg = spatial.grid_push_backward(V, T, G, b, o, ex)
    ran()
    ri, rg = O.grid_push_backward(vol, tgt, grid, [bound], [order], ex)
    assert relerr(np64(gi), ri) < tol and relerr(np64(gg), rg) < 1e-5
    gg = spatial.grid_count_backward(torch.ones_like(V[:, :1]).float(), G, b, o, ex)
    ran()
    assert relerr(np64(gg), O.grid_count_backward(np.ones_like(vol[:, :1]), grid, [bound], [order], ex)) < 1e-5


@pytest.mark.parametrize("lattice", SHAPES_3D)
@pytest.mark.parametrize("C", [1, 3, 6])
@pytest.mark.parametrize("bound,ex", [(7, 0), (2, 1), (3, 1)])
def test_linear_3d_tile_edges(lattice, C, bound, ex):
    _check(*_case(lattice, (6, 7, 11), C, 2, C + sum(lattice)), bound, 1, ex)


@pytest.mark.parametrize("lattice", SHAPES_3D)
@pytest.mark.parametrize("bound,ex", [(7, 0), (2, 1), (3, 1)])
def test_quadratic_3d_tile_edges(lattice, bound, ex):
    _check(*_case(lattice, (6, 7, 11), 1, 2, 2 + sum(lattice)), bound, 2, ex)


@pytest.mark.parametrize("lattice", SHAPES_2D)
@pytest.mark.parametrize("C", [2, 5])
@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("bound,ex", [(7, 1), (5, 0), (0, 1)])
def test_2d_tile_edges(lattice, C, order, bound, ex):
    _check(*_case(lattice, (13, 9), C, 3, C + order + sum(lattice)), bound, order, ex)


@pytest.mark.parametrize("dim,order", [(3, 1), (2, 3)])
def test_bfloat16(dim, order):
    lattice = (5, 9, 33)[:dim] if dim == 3 else (21, 35)
    vol, grid, tgt = _case(lattice, (6, 7, 11)[:dim], 3, 2, 5)
    _check(vol, grid, tgt, 2, order, 1, torch.bfloat16, 2.0 ** -8 + 1e-5)


def test_linear_3d_runs_of_planes():
    """Enough tiles for several planes per thread (3 x 5 tiles x 2 x 250
    planes over 148 * 8), the planes of an item no multiple of the run."""
    vol, grid, tgt = _case((250, 40, 70), (61, 23, 35), 1, 2, 3)
    _check(vol, grid, tgt, 2, 1, 1)


def test_strided_and_broadcast():
    """Channel-last images, an expanded (stride 0) batch of the grid and a
    strided target against the same call on contiguous copies."""
    vol, grid, tgt = _case((6, 9, 34), (7, 8, 9), 3, 2, 11)
    b, o = enums(5, 1)
    V = cu(vol, torch.float32).permute(0, 2, 3, 4, 1).contiguous().permute(0, 4, 1, 2, 3).requires_grad_()
    G = cu(grid[:1], torch.float32).expand(2, -1, -1, -1, -1).requires_grad_()
    T = cu(np.repeat(tgt, 2, -1), torch.float32)[..., ::2]
    Vc, Gc, Tc = (t.detach().contiguous().requires_grad_() for t in (V, G, T))
    for fn in (lambda v, g, t: [spatial.grid_pull(v, g, b, o, 1)],
               lambda v, g, t: [spatial.grid_push(t, g, [7, 8, 9], b, o, 1)],
               lambda v, g, t: spatial.grid_pull_backward(t, v, g, b, o, 1)):
        for got, ref in zip(fn(V, G, T), fn(Vc, Gc, Tc)):
            assert _lib.last_kernel().startswith("pp_direct_kernel")
            assert relerr(np64(got), np64(ref)) < 1e-6

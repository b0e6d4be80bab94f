"""The marching kernel of 3-D float32 displacement grids (solve.
c_regulariser_grid) against the FP64 oracle where its tiling can go wrong:
axes of one voxel and around the tile's extents, several chunks along the
marched axis, every stencil instance (radius 1 and 2, with and without the
Lame terms), Hessian layouts, bounds of either sign, batches, strided
fields.  Tolerance: float32 arithmetic, 1e-5 of max |ref|."""
import numpy as np
import pytest
import torch

from nitorch_b200 import solve
from oracle import oracle as O
from tests._gpu_ops import np64, relerr

pytestmark = pytest.mark.gpu

PENALTIES = [dict(absolute=0.1, membrane=0.7), dict(absolute=0.2, lame=(0.3, 0.5)),
             dict(absolute=0.1, bending=0.4), dict(absolute=0.1, membrane=0.3, bending=0.2, lame=(0.05, 0.2))]
CODES = {"dct2": 2, "dft": 5, "dst2": 4, "zero": 7, "dct1": 1}


def _run(v, hess, pen, bound, vs):
    pen = dict(pen)
    shear, div = pen.pop("lame", (0.0, 0.0))
    ref = O.regulariser_grid(np.moveaxis(np64(v), -1, 1), None, None if hess is None else np.moveaxis(np64(hess), -1, 1),
                             shear=shear, div=div, voxel_size=vs, bound=[CODES[b] for b in bound], **pen)
    out = solve.c_regulariser_grid(v, None, hess, lame=(shear, div), voxel_size=list(vs), bound=list(bound), **pen)
    assert relerr(np64(out), np.moveaxis(ref, 1, -1)) < 1e-5


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 8, 32), (9, 7, 31), (17, 9, 33), (40, 17, 5), (5, 16, 65)])
@pytest.mark.parametrize("pen", range(len(PENALTIES)))
@pytest.mark.parametrize("bound", [("dct2",) * 3, ("dft", "dst2", "zero"), ("dct1", "dft", "dst2")])
def test_tile_edges(shape, pen, bound):
    g = torch.Generator(device="cuda").manual_seed(pen + sum(shape))
    v = torch.randn((2, *shape, 3), generator=g, device="cuda")
    _run(v, None, PENALTIES[pen], bound, (1.0, 1.5, 0.8))


@pytest.mark.parametrize("DD", [1, 3, 6])
def test_hessians(DD):
    g = torch.Generator(device="cuda").manual_seed(DD)
    v = torch.randn((2, 11, 9, 34, 3), generator=g, device="cuda")
    h = torch.rand((2, 11, 9, 34, DD), generator=g, device="cuda")
    for pen in PENALTIES:
        _run(v, h, pen, ("dft",) * 3, (1.0, 1.0, 1.0))


def test_components_first_field():
    g = torch.Generator(device="cuda").manual_seed(3)
    v = torch.randn((1, 3, 12, 10, 35), generator=g, device="cuda").movedim(1, -1)
    _run(v, None, PENALTIES[3], ("dct2", "dft", "dct2"), (1.0, 1.0, 1.0))

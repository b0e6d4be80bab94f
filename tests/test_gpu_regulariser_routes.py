"""Which kernel regularises a 3-D float32 displacement grid: the marching one
where its columns of 8 x 32 voxels are mostly inside the volume and there are
enough of them, one thread per voxel elsewhere; both against the FP64 oracle at
sizes next to the line.  Tolerance: float32 arithmetic, 1e-5 of max |ref|."""
import numpy as np
import pytest
import torch

from nitorch_b200 import _lib, solve
from oracle import oracle as O
from tests._gpu_ops import np64, relerr

pytestmark = pytest.mark.gpu

TERMS = {"membrane": dict(absolute=0.1, membrane=0.7), "lame": dict(absolute=0.2, lame=(0.3, 0.5)),
         "bending": dict(absolute=0.1, bending=0.4),
         "all": dict(absolute=0.1, membrane=0.3, bending=0.2, lame=(0.05, 0.2))}
CODES = {"dct2": 2, "dft": 5, "dst2": 4, "zero": 7, "dct1": 1}


def _check(terms, shape, kernel, bound, DD=None):
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    v = torch.randn((2, *shape, 3), generator=g, device="cuda")
    h = torch.rand((2, *shape, DD), generator=g, device="cuda") if DD else None
    pen = dict(TERMS[terms])
    shear, div = pen.pop("lame", (0.0, 0.0))
    vs = (1.0, 1.5, 0.8)
    out = solve.c_regulariser_grid(v, None, h, lame=(shear, div), voxel_size=list(vs), bound=list(bound), **pen)
    assert _lib.last_kernel().startswith(kernel + " "), _lib.last_kernel()
    ref = O.regulariser_grid(np.moveaxis(np64(v), -1, 1), None, None if h is None else np.moveaxis(np64(h), -1, 1),
                             shear=shear, div=div, voxel_size=vs, bound=[CODES[b] for b in bound], **pen)
    assert relerr(np64(out), np.moveaxis(ref, 1, -1)) < 1e-5


@pytest.mark.parametrize("terms,shape", [("membrane", (33, 41, 65)), ("membrane", (25, 260, 11)), ("lame", (20, 25, 70)),
                                         ("bending", (9, 17, 33)), ("all", (9, 17, 33)), ("all", (70, 16, 7))])
@pytest.mark.parametrize("bound", [("dct2",) * 3, ("dft", "dst2", "zero"), ("dct1", "dft", "dst2")])
def test_marching(terms, shape, bound):
    _check(terms, shape, "regulariser_march_kernel", bound)


@pytest.mark.parametrize("DD", [1, 3, 6])
def test_marching_hessians(DD):
    for terms, shape in (("all", (9, 17, 33)), ("membrane", (33, 41, 65))):
        _check(terms, shape, "regulariser_march_kernel", ("dft",) * 3, DD)


@pytest.mark.parametrize("terms,shape", [("membrane", (80, 120, 8)), ("membrane", (32, 32, 32)), ("lame", (50, 64, 6)),
                                         ("lame", (24, 24, 24)), ("bending", (40, 64, 5)), ("bending", (14, 14, 14)),
                                         ("all", (40, 64, 4)), ("all", (200, 3, 1))])
def test_thin_and_small(terms, shape):
    _check(terms, shape, "regulariser_kernel", ("dct2", "dft", "dct1"))

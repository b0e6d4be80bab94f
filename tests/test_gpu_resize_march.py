"""The marching form of the separable resize (pp_resize) on volumes with
several columns and chunks: columns inside the volume (TMA copies) beside
columns at its edges, every tile the steps select, several chunks along x,
the steps around the limit where the tiled form takes over, bfloat16 and
channel-last images.  Against the per-point affine pull of the same map at
1e-6 of max |ref| (float32 rounding of differently ordered sums), bfloat16
within one storage rounding."""
import numpy as np
import pytest
import torch

from nitorch_b200 import _lib, affine
from nitorch_b200.enums import BoundType
from tests._gpu_ops import np64, relerr

pytestmark = pytest.mark.gpu


def _both(x, scales, shifts, shape, order, bound, ex):
    mat = torch.zeros((x.shape[0], 3, 4))
    for d in range(3):
        mat[:, d, d], mat[:, d, 3] = scales[d], shifts[d]
    out = affine.resize_pull(x, scales, shifts, shape, order, BoundType(bound), ex)
    kern = _lib.last_kernel()
    ref = affine.affine_pull(x, mat.cuda(), shape, order, BoundType(bound), ex)
    assert affine.resize_status() == 0
    return np64(out), np64(ref), kern


@pytest.mark.parametrize("order", [0, 1, 2, 3])
@pytest.mark.parametrize("bound", [2, 5, 3, 7])
@pytest.mark.parametrize("scales,shape", [
    ((0.8, 0.8, 0.8), (150, 75, 210)),    # 32 x 64 tiles
    ((0.4, 1.2, 0.9), (90, 60, 140)),     # 16 x 64 or 8 x 64 tiles
    ((2.1, 1.9, 2.2), (20, 31, 70)),      # 8 x 32 tiles
    ((1.0, 2.6, 2.6), (33, 30, 60)),      # past the marching form's steps for cubic stencils
])
def test_columns_and_chunks(order, bound, scales, shape):
    g = torch.Generator().manual_seed(order + 10 * bound)
    inshape = tuple(int(s * o) + 3 for s, o in zip(scales, shape))
    x = torch.randn((1, 2, *inshape[:2], (inshape[2] + 3) // 4 * 4), generator=g).cuda()
    out, ref, kern = _both(x, scales, (-0.6, 0.3, 0.2), shape, order, bound, 0)
    assert "tma" in kern and ("march" in kern or scales[1] > 2.5), kern
    assert not ("march" in kern and scales[1] > 2.5 and order == 3), kern
    assert relerr(out, ref) < 1e-6


@pytest.mark.parametrize("shape", [(1, 1, 1), (9, 8, 32), (65, 33, 65)])
def test_ragged_outputs(shape):
    x = torch.randn((2, 1, 17, 30, 60), generator=torch.Generator().manual_seed(1)).cuda()
    out, ref, _ = _both(x, (0.3, 0.9, 0.9), (0.1, -1.3, 2.4), shape, 3, 2, 1)
    assert relerr(out, ref) < 1e-6


def test_bfloat16_and_channel_last():
    x = torch.randn((1, 40, 60, 120, 3), generator=torch.Generator().manual_seed(2)).cuda().movedim(-1, 1)
    out, ref, kern = _both(x, (0.8,) * 3, (0.1,) * 3, (48, 70, 145), 3, 2, 0)
    assert "march" in kern and "tma" not in kern and relerr(out, ref) < 1e-6
    out, ref, kern = _both(x.contiguous().bfloat16(), (0.8,) * 3, (0.1,) * 3, (48, 70, 145), 3, 2, 0)
    assert "march" in kern and relerr(out, ref) < 2.0 ** -8

"""The prefilter's lines cut into segments, against the FP64 oracle where the
cut can go wrong: lengths at which the number of segments or of lines per tile
changes (a segment is longer than its warm-up of ceil(-30 / ln|z|) samples),
segments of unequal length, tiles with missing lines, and lines read in groups
of four next to lines that are not aligned for it.  Tolerances: float32
recursions 1e-5, one bfloat16 rounding of the output 8e-3."""
import math

import numpy as np
import pytest
import torch

from nitorch_b200 import coeff
from oracle import oracle as O
from tests._gpu_ops import relerr

pytestmark = pytest.mark.gpu

POLE = {2: math.sqrt(8) - 3, 3: math.sqrt(3) - 2, 7: -0.5352804307964382}


def _lengths(order):
    w = math.ceil(-30 / math.log(-POLE[order])) + 1
    return [2 * w - 1, 2 * w, 4 * w - 1, 4 * w, 4 * w + 3, 415, 416, 803, 804]


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 8e-3)])
@pytest.mark.parametrize("bound", [2, 3, 6])
@pytest.mark.parametrize("order", sorted(POLE))
def test_segment_edges(order, bound, dtype, tol):
    r = np.random.default_rng(order + bound)
    for n in _lengths(order):
        for shape, axis in (((67, n), -1), ((n, 68), 0)):
            x = torch.from_numpy(r.standard_normal(shape)).to(dtype)
            ref = O.spline_coeff(x.double().numpy(), bound, order, dim=axis)
            X = x.cuda()
            assert relerr(coeff.spline_coeff(X, bound, order, dim=axis).double().cpu().numpy(), ref) < tol
            Y = torch.empty(X.numel() + 1, dtype=dtype, device="cuda")[1:].view(shape)  # off the alignment
            Y.copy_(X)
            out = coeff.spline_coeff(Y, bound, order, dim=axis, inplace=True)
            assert out.data_ptr() == Y.data_ptr()
            assert relerr(Y.double().cpu().numpy(), ref) < tol

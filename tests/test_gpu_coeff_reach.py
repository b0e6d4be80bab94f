"""How far a sample reaches along a prefiltered line that is cut into segments:
as far as along a whole one.  A NaN, an infinity and a sample of 1e25 among
samples of unit scale, and a block of samples among exact zeros, in every
segment of a line, against the same call on float64 lines, which are never cut.
Finite values: float32 rounding of the recursions, 1e-5 of the envelope
max_k |ref[k]| |z|^|i - k| (what a coefficient is summed from; around the ends
of a periodic line)."""
import math

import numpy as np
import pytest
import torch

from nitorch_b200 import coeff

pytestmark = pytest.mark.gpu

POLE = {2: math.sqrt(8) - 3, 3: math.sqrt(3) - 2, 7: -0.5352804307964382}


def _envelope(ref, z, periodic):
    n = ref.shape[1]
    env = np.abs(np.tile(ref, 3) if periodic else ref)
    for order in (range(1, env.shape[1]), range(env.shape[1] - 2, -1, -1)):
        step = 1 if order.step > 0 else -1
        for i in order:
            env[:, i] = np.maximum(env[:, i], env[:, i - step] * z)
    return env[:, n:2 * n] if periodic else env


def _lines(kind, n, r):
    x = r.standard_normal((66, n)).astype(np.float32)
    for line, at in enumerate(np.linspace(0, n - 1, 66).astype(int)):
        if kind == "block":
            keep = x[line, at:at + 3].copy()
            x[line] = 0
            x[line, at:at + 3] = keep
        else:
            x[line, at] = {"nan": np.nan, "inf": -np.inf, "huge": 1e25}[kind]
    return x


@pytest.mark.parametrize("kind", ["nan", "inf", "huge", "block"])
@pytest.mark.parametrize("bound", [2, 3, 6])
@pytest.mark.parametrize("order", sorted(POLE))
def test_reach(order, bound, kind):
    r = np.random.default_rng(7)
    for n in (256, 415):
        x = _lines(kind, n, r)
        ref = coeff.spline_coeff(torch.from_numpy(x).double().cuda(), bound, order).cpu().numpy()
        for axis in (-1, 0):
            X = torch.from_numpy(x if axis else np.ascontiguousarray(x.T)).cuda()
            out = coeff.spline_coeff(X, bound, order, dim=axis).double().cpu().numpy()
            out = out if axis else out.T
            assert (np.isnan(out) == np.isnan(ref)).all()
            inf = np.isinf(ref)
            assert (np.isinf(out) == inf).all() and (out[inf] == ref[inf]).all()
            fin = np.isfinite(ref).all(1)
            env = _envelope(ref[fin], -POLE[order], bound == 6)
            assert (np.abs(out[fin] - ref[fin]) <= 1e-5 * env + 1e-38).all()


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 8e-3)])
@pytest.mark.parametrize("lines", [28416, 28417, 30001, 37888, 37889])
def test_many_lines(lines, dtype, tol):
    """Line counts around one wave of 128-line tiles (two segments per line)."""
    g = torch.Generator(device="cuda").manual_seed(lines)
    x = torch.randn(lines, 200, device="cuda", generator=g).to(dtype)
    x[::1000, 61] = float("nan")
    ref = coeff.spline_coeff(x.double(), 3, 3)
    for axis in (-1, 0):
        out = coeff.spline_coeff(x if axis else x.T.contiguous(), 3, 3, dim=axis).double()
        out = out if axis else out.T
        assert torch.equal(out.isnan(), ref.isnan())
        assert float((out - ref).nan_to_num().abs().max() / ref.nan_to_num().abs().max()) < tol

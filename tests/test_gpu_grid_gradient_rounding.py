"""Rounding of the direct kernels' grid gradients of several channels: no larger
than that of the plain float32 sums in which every channel's differences are
formed by themselves and multiplied by the incoming gradient afterwards (torch
on the CPU, each operation rounded; the kernel's fused operations round less
often).  RMS errors against the same sums in float64, margin 1.1."""
import pytest
import torch

from nitorch_b200 import _lib, spatial
from tests._gpu_ops import enums

pytestmark = pytest.mark.gpu


def _plain(image, target, grid, dtype):
    """Linear grid gradient inside the volume: sum_c t_c grad(image_c)."""
    dim = grid.shape[-1]
    x, g = image[0].to(dtype), grid[0].to(dtype)
    fl = g.floor()
    f = g - fl
    lo = [fl[..., d].long() for d in range(dim)]
    w = [(1 - f[..., d], f[..., d]) for d in range(dim)]
    out = []
    for d in range(dim):

        def total(axis, idx):  # first axis innermost, as the kernels sum
            if axis < 0:
                return x[(slice(None), *idx)]
            parts = [total(axis - 1, [lo[axis] + k, *idx]) for k in (0, 1)]
            if axis == d:
                return parts[1] - parts[0]
            return w[axis][0] * parts[0] + w[axis][1] * parts[1]

        rows = total(dim - 1, [])
        s = target[0, 0].to(dtype) * rows[0]
        for c in range(1, x.shape[0]):
            s = s + target[0, c].to(dtype) * rows[c]
        out.append(s)
    return torch.stack(out, -1)


@pytest.mark.parametrize("dim,C,op", [(2, 2, "pull"), (2, 4, "pull"), (2, 8, "pull"), (2, 4, "push"), (3, 4, "push"),
                                      (3, 3, "push"), (3, 6, "pull")])
def test_rounding(dim, C, op):
    g = torch.Generator().manual_seed(dim + C)
    size = (200, 170) if dim == 2 else (31, 37, 41)
    # smooth images, as volumes are: neighbouring values nearly cancel
    axes = torch.meshgrid(*[torch.arange(float(s)) for s in size], indexing="ij")
    wave = torch.randn(C, dim + 1, generator=g) * 0.1
    image = torch.stack([torch.cos(sum(w[d] * axes[d] for d in range(dim)) + 10 * w[-1]) for w in wave])[None]
    target = torch.randn(1, C, *size, generator=g)
    grid = torch.rand(1, *size, dim, generator=g) * torch.tensor([s - 1.001 for s in size])
    ref = _plain(image, target, grid, torch.float64)
    plain = _plain(image, target, grid, torch.float32).double()
    b, o = enums(2, 1)
    if op == "pull":
        out = spatial.grid_pull_backward(target.cuda(), image.cuda().requires_grad_(), grid.cuda().requires_grad_(), b, o, 1)
    else:
        out = spatial.grid_push_backward(image.cuda(), target.cuda().requires_grad_(), grid.cuda().requires_grad_(), b, o, 1)
    assert _lib.last_kernel().startswith("pp_direct_kernel")
    err = (out[1][0].double().cpu() - ref).pow(2).mean().sqrt()
    assert err <= 1.1 * (plain - ref).pow(2).mean().sqrt()

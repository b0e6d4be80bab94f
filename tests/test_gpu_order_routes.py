"""Calls of the direct kernels' stencils that are given a sample order, or that
the direct kernels refuse by size: the kernels that use the order run, with the
natural order's results (tolerance: float32 summation order, 1e-5)."""
import pytest
import torch

from nitorch_b200 import _lib, spatial
from tests._gpu_ops import enums

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _restore():
    yield
    spatial.set_sample_order("auto")


def _calls(size, src, order, channels=2):
    g = torch.Generator(device="cuda").manual_seed(1)
    dim = len(size)
    grid = torch.rand(1, *size, dim, device="cuda", generator=g) * torch.tensor([s - 1. for s in src], device="cuda")
    image = torch.randn(1, channels, *src, device="cuda", generator=g).requires_grad_()
    values = torch.randn(1, channels, *size, device="cuda", generator=g)
    b, o = enums(2, order)
    out, kernels = [], []
    for f in (lambda: [spatial.grid_pull(image, grid, b, o, 1)], lambda: [spatial.grid_grad(image, grid, b, o, 1)],
              lambda: [spatial.grid_push(values, grid, list(src), b, o, 1)],
              lambda: [spatial.grid_pull_backward(values, image, grid, b, o, 1)[0]]):
        out += f()
        kernels.append(_lib.last_kernel())
    return out, kernels


@pytest.mark.parametrize("size,src,order", [((20, 31, 33), (15, 16, 17), 1), ((90, 70), (40, 50), 1), ((90, 70), (40, 50), 3)])
def test_given_order_is_used(size, src, order):
    spatial.set_sample_order("natural")
    ref, kernels = _calls(size, src, order)
    assert all(k.startswith("pp_direct_kernel") for k in kernels), kernels
    spatial.set_sample_order("sorted")
    out, kernels = _calls(size, src, order)
    assert not any(k.startswith("pp_direct_kernel") for k in kernels), kernels
    for a, r in zip(out, ref):
        assert float((a - r).abs().max() / r.abs().max()) < 1e-5


def test_refused_sizes_keep_their_order(monkeypatch):
    """A middle axis of more tiles than a launch has, 2^18 points and more."""
    spatial.set_sample_order("natural")
    ref, _ = _calls((70000, 4), (300, 200), 1)
    spatial.set_sample_order("auto")
    orders = []
    made = spatial.sample_order
    monkeypatch.setattr(spatial, "sample_order", lambda *a: orders.append(made(*a)) or orders[-1])
    out, kernels = _calls((70000, 4), (300, 200), 1)
    assert len(orders) == 1 and not any(k.startswith("pp_direct_kernel") for k in kernels)
    for a, r in zip(out, ref):
        assert float((a - r).abs().max() / r.abs().max()) < 1e-5


@pytest.mark.parametrize("n,order,bricks", [(66, 3, (True, False, True, True)), (66, 2, (False, False, False, False)),
                                            (84, 3, (True, True, True, True)), (84, 2, (True, True, False, False))])
def test_small_volumes_run_per_point(n, order, bricks):
    """Ordered grids of 2^18 points and more whose windows do not pay."""
    spatial.set_sample_order("natural")
    ref, _ = _calls((n, n, n), (n, n, n), order)
    spatial.set_sample_order("auto")
    out, kernels = _calls((n, n, n), (n, n, n), order)
    assert tuple(k.startswith("pp_brick_") for k in kernels) == bricks, kernels
    assert not any(k.startswith("pp_direct_") for k in kernels), kernels
    for a, r in zip(out, ref):
        assert float((a - r).abs().max() / r.abs().max()) < 1e-5


@pytest.mark.parametrize("order", [2, 3])
def test_rounding_does_not_depend_on_the_order(order):
    """RMS error against float64 of the gathers that small volumes leave to the
    per-point kernel: no larger than the brick kernels' (the same weights; sums
    in another order: margin 1.1)."""
    g = torch.Generator(device="cuda").manual_seed(order)
    image = torch.rand(1, 3, 40, 41, 42, device="cuda", generator=g).requires_grad_()
    grid = (torch.rand(1, 60, 61, 62, 3, device="cuda", generator=g) * 38 + 1).requires_grad_()
    target = torch.rand(1, 3, 60, 61, 62, device="cuda", generator=g)
    b, o = enums(2, order)

    def run(dt):
        x, p, t = (v.detach().to(dt).requires_grad_() for v in (image, grid, target))
        return [spatial.grid_pull(x, p, b, o, 1), spatial.grid_grad(x, p, b, o, 1), *spatial.grid_push_backward(x.detach(), t, p, b, o, 1)]

    errors = {}
    ref = run(torch.float64)
    for mode in ("natural", "sorted"):
        spatial.set_sample_order(mode)
        out = run(torch.float32)
        assert _lib.last_kernel().startswith("pp_brick_" if mode == "sorted" else ("pp_direct", "pp_kernel", "pp_lanes"))
        errors[mode] = [float((a.double() - r).pow(2).mean().sqrt()) for a, r in zip(out, ref)]
    for a, r in zip(errors["natural"], errors["sorted"]):
        assert a <= 1.1 * r, errors

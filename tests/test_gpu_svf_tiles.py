"""The linear self-composition kernels of velocity exponentiation (3-D
float32) against the FP64 oracle where their tiles and the sums shared by
neighbouring voxels can go wrong: axes of one voxel and around a tile's 8 x 32
voxels, runs of planes across batch items, smooth fields (cells that follow
one another along x and z), rough fields, constant shifts past the edge,
every bound, four-slot and strided layouts.  Tolerance: float32 1e-5 of
max |ref|."""
import numpy as np
import pytest
import torch

from nitorch_b200 import _lib, svf
from oracle import oracle as O
from tests._gpu_ops import np64, relerr

pytestmark = pytest.mark.gpu

NAMES = {0: "replicate", 1: "dct1", 2: "dct2", 3: "dst1", 4: "dst2", 5: "dft", 7: "zero"}


def _field(shape, kind, seed, N=3):
    r = np.random.default_rng(seed)
    if kind == "rough":
        return 2.5 * r.standard_normal((N, *shape, 3))
    if kind == "shift":  # whole voxels and a fraction, past the edges
        return np.broadcast_to(r.uniform(-3.0, 3.0, (N, 1, 1, 1, 3)), (N, *shape, 3)).copy()
    mesh = np.stack(np.meshgrid(*[np.linspace(0, 3, s) for s in shape], indexing="ij"), -1)
    return 0.4 * np.sin(mesh[None] + r.uniform(0, 6, (N, 1, 1, 1, 3)))


def _layout(a, four):
    t = torch.as_tensor(a, dtype=torch.float32, device="cuda")
    if not four:
        return t.contiguous()
    out = torch.empty((*t.shape[:-1], 4), device="cuda")[..., :3]
    return out.copy_(t)


@pytest.mark.parametrize("shape", [(1, 1, 1), (5, 9, 33), (7, 8, 32), (4, 17, 3), (40, 3, 70)])
@pytest.mark.parametrize("kind", ["smooth", "rough", "shift"])
@pytest.mark.parametrize("bound", sorted(NAMES))
@pytest.mark.parametrize("ex", [0, 1])
def test_tiles(shape, kind, bound, ex):
    seed = sum(shape) + bound
    u = _field(shape, kind, seed).astype(np.float32).astype(np.float64)
    g = np.random.default_rng(seed + 1).standard_normal(u.shape).astype(np.float32).astype(np.float64)
    ref = O.svf_compose(u, bound, 1, ex)
    rbk = O.svf_compose_backward(g, u, bound, 1, ex)
    for four in (False, True):
        U, G = _layout(u, four), _layout(g, four)
        out = svf.compose(U, "linear", NAMES[bound], ex)
        assert _lib.last_kernel().startswith("svf_compose_lin3")
        assert relerr(np64(out), ref) < 1e-5
        back = svf.compose_backward(G, U, "linear", NAMES[bound], ex, deterministic=False)
        assert _lib.last_kernel().startswith("svf_compose_backward_lin3")
        assert relerr(np64(back), rbk) < 1e-5

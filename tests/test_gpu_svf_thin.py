"""The linear self-composition kernels on planes that their tiles cover in
other proportions than 8 x 32: short axes and axes next to a tile's extent, with
cells that follow one another from one row of a tile to the next.  Against the
FP64 oracle, float32 1e-5 of max |ref|."""
import numpy as np
import pytest

from nitorch_b200 import _lib, svf
from oracle import oracle as O
from tests._gpu_ops import np64, relerr
from tests.test_gpu_svf_tiles import NAMES, _field, _layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 300, 1), (3, 129, 2), (5, 65, 3), (4, 40, 8), (3, 17, 9), (3, 9, 16), (3, 20, 40),
                                   (4, 4, 65), (3, 2, 129), (3, 1, 257)])
@pytest.mark.parametrize("kind", ["smooth", "rough", "shift"])
@pytest.mark.parametrize("bound", [2, 5, 7])
def test_thin(shape, kind, bound):
    seed = sum(shape) + bound
    # multiples of 2^-12: voxel index + displacement is exact in float32, as the oracle has it
    u = np.round(_field(shape, kind, seed, 2) * 4096) / 4096
    g = np.random.default_rng(seed + 1).standard_normal(u.shape).astype(np.float32).astype(np.float64)
    for four in (False, True):
        U, G = _layout(u, four), _layout(g, four)
        out = svf.compose(U, "linear", NAMES[bound], 1)
        assert _lib.last_kernel().startswith("svf_compose_lin3")
        assert relerr(np64(out), O.svf_compose(u, bound, 1, 1)) < 1e-5
        back = svf.compose_backward(G, U, "linear", NAMES[bound], 1, deterministic=False)
        assert relerr(np64(back), O.svf_compose_backward(g, u, bound, 1, 1)) < 1e-5

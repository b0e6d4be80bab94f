"""The direct kernels on grids that their tiles cover in other proportions than
8 x 32: axes of one to three points beside long ones, next to a tile's extent.
Tolerances as in test_gpu_direct.py."""
import pytest

from tests.test_gpu_direct import _case, _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice", [(4, 300, 2), (3, 129, 1), (3, 90, 4), (3, 2, 300), (2, 1, 257), (2, 4, 70)])
@pytest.mark.parametrize("C", [1, 3])
@pytest.mark.parametrize("bound,ex", [(7, 0), (2, 1)])
def test_3d(lattice, C, bound, ex):
    _check(*_case(lattice, (6, 7, 11), C, 2, C + sum(lattice)), bound, 1, ex)


@pytest.mark.parametrize("lattice", [(300, 2), (257, 1), (70, 3), (2, 300), (1, 257), (3, 130)])
@pytest.mark.parametrize("order", [1, 2, 3])
def test_2d(lattice, order):
    _check(*_case(lattice, (13, 9), 2, 3, order + sum(lattice)), 2, order, 1)

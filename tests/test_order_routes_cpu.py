"""Which calls leave their points in the grid's own order: those that the
direct kernels take, within the sizes that they take (meta tensors: no data)."""
import pytest
import torch

from nitorch_b200 import spatial


def _grid(*size, dtype=torch.float32):
    return torch.empty(*size, len(size) - 1, device="meta", dtype=dtype)


def _image(*size, dtype=torch.float32):
    return torch.empty(*size, device="meta", dtype=dtype)


def _direct(grid, order, image, src=(64, 64, 64)):
    dim = grid.dim() - 2
    return spatial._direct(grid, src[:dim], [order] * dim, (image,))


@pytest.mark.parametrize("order,channels,expected", [(1, 1, True), (1, 5, True), (2, 1, True), (2, 2, False), (3, 1, False)])
def test_orders(order, channels, expected):
    assert _direct(_grid(1, 64, 64, 64), order, _image(1, channels, 64, 64, 64)) is expected


def test_sizes():
    image3, image2 = _image(1, 1, 64, 64, 64), _image(1, 1, 64, 64)
    assert _direct(_grid(1, 2, 65535, 4), 1, image3)
    assert not _direct(_grid(1, 2, 65536, 4), 1, image3)          # tiles along the middle axis
    assert _direct(_grid(1, 65535, 8), 3, image2)
    assert not _direct(_grid(1, 70000, 4), 3, image2)
    assert not _direct(_grid(4, 1 << 22, 2, 2), 1, image3)        # planes
    assert not _direct(_grid(1, 900, 900, 900), 1, image3)        # grid offsets
    assert not _direct(_grid(1, 64, 64, 64), 1, _image(1, 4, 900, 900, 900), (900,) * 3)
    assert not _direct(_grid(1, 64, 64, 64), 1, image3, (1300,) * 3)
    sliced = _image(1, 1, 1300, 1300, 1300)[..., ::20, ::20, ::20]
    assert not _direct(_grid(1, 64, 64, 64), 1, sliced)           # strides count, not elements


def test_types():
    image = _image(1, 1, 64, 64, 64)
    assert _direct(_grid(1, 64, 64, 64), 1, image.to(torch.bfloat16))
    assert not _direct(_grid(1, 64, 64, 64), 1, image.to(torch.float16))
    assert not _direct(_grid(1, 64, 64, 64, dtype=torch.float64), 1, image.double())

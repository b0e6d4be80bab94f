"""Bounds and orders are read anew from objects that may change between calls:
only names, integers and enum members are remembered."""
import pytest
import torch

from nitorch_b200.enums import BoundType, InterpolationType
from nitorch_b200.grid import _opt


def test_tensor_order_changed_in_place():
    order = torch.tensor(1)
    assert _opt("dct2", order, 0)[1] == [InterpolationType.linear]
    order.fill_(3)
    assert _opt("dct2", order, 0)[1] == [InterpolationType.cubic]


@pytest.mark.parametrize("order", [1, "linear", InterpolationType.linear, 1.0])
@pytest.mark.parametrize("bound", ["dct2", "reflect", BoundType.dct2])
def test_spellings(bound, order):
    for _ in range(2):
        b, o, ex = _opt([bound, "dft"], [order], True)
        assert b == [BoundType.dct2, BoundType.dft] and o == [InterpolationType.linear] and ex == 1
        b.append(None)
        o.append(None)  # a caller's list is its own


def test_refused():
    for _ in range(2):
        for bound, order in (("dct2", 8), ("nope", 1), (2, 1), ("dct2", "tenth")):
            with pytest.raises(ValueError):
                _opt(bound, order, 0)

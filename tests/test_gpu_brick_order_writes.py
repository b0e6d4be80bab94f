"""The brick order of a grid that another stream writes meanwhile is some
order: every sample once, brick offsets within the samples."""
import pytest
import torch

from nitorch_b200 import spatial

pytestmark = pytest.mark.gpu


def test_grid_written_while_it_is_ordered():
    size = (96, 90, 100)
    n = size[0] * size[1] * size[2]
    grid = torch.rand(1, *size, 3, device="cuda") * 90
    flat = grid.view(-1)
    other = torch.cuda.Stream()
    other.wait_stream(torch.cuda.current_stream())
    orders = []
    for _ in range(20):
        with torch.cuda.stream(other):
            for _ in range(10):
                flat.uniform_(0, 90)
        orders.append(spatial.brick_order(grid, size))
    torch.cuda.synchronize()
    every = torch.arange(n, dtype=torch.int32, device="cuda")
    for perm, starts, records in orders:
        assert torch.equal(perm.sort().values, every)
        assert int(starts[0]) == 0 and int(starts[-1]) == n and bool((starts[1:] >= starts[:-1]).all())
        assert torch.equal(records[:, 3].contiguous().view(torch.int32), perm)

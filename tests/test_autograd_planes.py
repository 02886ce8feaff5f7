"""The plane addresses that the autograd passes hand to the library against those of the tensor's views: rows longer
than the splat count, more than three rows, other element sizes; fewer than three rows are refused."""
import pytest
import torch

from splatter_gb300.autograd import _planes


@pytest.mark.parametrize("shape", [(3, 1), (3, 5), (3, 4096), (4, 7), (3, 2, 3), (3,)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_planes_are_the_rows(shape, dtype):
    t = torch.zeros(shape, dtype=dtype)
    assert _planes(t) == tuple(t[k].data_ptr() for k in range(3))


@pytest.mark.parametrize("shape", [(), (0, 4), (1, 4), (2, 4)])
def test_missing_planes_are_refused(shape):
    with pytest.raises(IndexError):
        _planes(torch.zeros(shape))

"""Views of the library's arrays: an array that the library does not have is an empty tensor, never memory of the asked
size."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ptr", [None, 0])
@pytest.mark.parametrize("shape", [5, (5,), (5, 3), 0, (0, 3)])
def test_an_absent_array_is_an_empty_view(cs, shape, ptr):
    t = cs._wrap(ptr, shape, torch.int32)
    assert t.numel() == 0 and t.dtype == torch.int32 and t.is_cuda
    assert t.dim() == (len(shape) if isinstance(shape, tuple) else 1) and t.shape[1:] == torch.Size(
        shape[1:] if isinstance(shape, tuple) else ())

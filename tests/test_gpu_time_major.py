"""The transposition between convolutions and recurrence (`csrc/cuda/transpose.cu`) against torch's permute, forward and backward, at the
edges of the 64 x 64 tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(32, 32, 41, 350), (1, 1, 1, 1), (3, 2, 32, 64), (2, 5, 13, 65), (5, 9, 7, 63), (7, 1, 1, 130), (2, 64, 2, 1)])
def test_matches_permute(shape):
    from tensorflow_allreduce_b200 import _lib

    torch.manual_seed(sum(shape))
    x = torch.randn(*shape, device="cuda", requires_grad=True)
    y = _lib.ext().time_major(x)
    want = x.detach().view(shape[0], -1, shape[-1]).permute(2, 0, 1)
    assert torch.equal(y, want) and y.is_contiguous()
    g = torch.randn_like(y)
    (dx,) = torch.autograd.grad(y, x, g)
    assert torch.equal(dx, g.permute(1, 2, 0).reshape(shape))

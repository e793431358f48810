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


def test_a_model_without_the_library_s_kernels_launches_none(monkeypatch):
    from tensorflow_allreduce_b200 import _lib
    from tensorflow_allreduce_b200.models import ds2

    cfg = ds2.DS2Config(n_frames=40, rnn_hidden=128, rnn_layers=1, label_len=5)
    off = ds2.DS2Config(**{**vars(cfg), "persistent_rnn": False, "fused_norm": False, "row_conv": False})
    torch.manual_seed(0)
    model, stock = ds2.DeepSpeech2(cfg).cuda(), ds2.DeepSpeech2(off).cuda()
    stock.load_state_dict(model.state_dict())
    spect = ds2.synthetic_batch(cfg, 4, "cuda")[0]
    want = model(spect)

    def refuse():
        raise AssertionError("the extension was asked for")

    monkeypatch.setattr(_lib, "ext", refuse)
    got = stock(spect)
    got.sum().backward()
    assert (got - want).norm().item() < 5e-3 * want.norm().item()

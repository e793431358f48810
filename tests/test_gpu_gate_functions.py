"""The gate functions of the persistent GRU kernels against fp64, one function at a time through the public entry point: with recurrent
weights of zero and an update gate of zero, the output of a step is the tanh of its input; a step whose candidate is zero after a step
whose output is one gives the sigmoid.

Errors are in units in the last place of the exact value. The limits are those of CUDA's `tanhf` and `1.f / (1.f + __expf(-x))` over ALL
floats of each range on a B200 (largest, mean): functions in their place may not be further off. A sample's mean differs from the mean over
all floats by less than 1 % (half a million values with a deviation of about their mean)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TANH = [(1e-30, 1e-3, 0.501, 0.0081), (1e-3, 0.1, 1.04, 0.2657), (0.1, 0.625, 1.81, 0.6343), (0.625, 1.0, 1.81, 0.3827), (1.0, 2.0, 1.38, 0.2768),
        (2.0, 9.0, 0.68, 0.2504), (9.0, 80.0, 0.501, 0.0103)]
SIGMOID = [(0.1, 0.625, 1.42, 0.3304), (1.0, 2.0, 1.60, 0.4183), (2.0, 9.0, 1.59, 0.5196), (9.0, 80.0, 1.26, 0.1666),
           (-0.1, -0.625, 2.40, 0.5540), (-1.0, -2.0, 3.46, 0.5333), (-2.0, -9.0, 8.44, 1.3367), (-9.0, -80.0, 62.3, 9.1599)]


def _floats(lo, hi, n):
    """n floats of [lo, hi), every representable one as likely."""
    a, b = torch.tensor([abs(lo), abs(hi)]).view(torch.int32).tolist()
    v = torch.randint(a, b, (n,), device="cuda", dtype=torch.int32).view(torch.float32)
    return v if lo > 0 else -v


def _run(gx):
    """gx [T, B, 3 * 128] as the input projections of a layer without recurrent weights; its outputs."""
    from tensorflow_allreduce_b200.ops import persistent_gru as pg

    rnn = torch.nn.GRU(384, 128).cuda()
    old = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    try:
        with torch.no_grad():
            for p in rnn.parameters():
                p.zero_()
            rnn.weight_ih_l0.copy_(torch.eye(384))
            y = pg.gru_forward(rnn, gx)
        pg.check_status()
        return y
    finally:
        torch.backends.cuda.matmul.allow_tf32 = old


def _units_off(got, want):
    unit = torch.ldexp(torch.ones_like(want), torch.frexp(want)[1].clamp(min=-125) - 24)
    return ((got.double() - want).abs() / unit)


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("lo,hi,largest,mean", TANH)
def test_tanh(lo, hi, largest, mean, sign):
    torch.manual_seed(0)
    x = _floats(sign * lo, sign * hi, 128 * 32 * 128).view(128, 32, 128)
    gx = torch.zeros(128, 32, 384, device="cuda")
    gx[..., 128:256] = -200.0
    gx[..., 256:] = x
    off = _units_off(_run(gx), torch.tanh(x.double()))
    print(f"tanh [{sign * lo}, {sign * hi}): {off.max().item():.3f} {off.mean().item():.4f}")
    assert off.max().item() <= largest and off.mean().item() <= 1.02 * mean + 1e-3


@pytest.mark.parametrize("lo,hi,largest,mean", SIGMOID)
def test_sigmoid(lo, hi, largest, mean):
    torch.manual_seed(0)
    x = _floats(lo, hi, 128 * 32 * 128).view(128, 32, 128)
    gx = torch.zeros(256, 32, 384, device="cuda")
    gx[0::2, :, 128:256] = -200.0
    gx[0::2, :, 256:] = 50.0
    gx[1::2, :, 128:256] = x
    y = _run(gx)
    assert (y[0::2] == 1).all()
    off = _units_off(y[1::2], torch.sigmoid(x.double()))
    print(f"sigmoid [{lo}, {hi}): {off.max().item():.3f} {off.mean().item():.4f}")
    assert off.max().item() <= largest and off.mean().item() <= 1.02 * mean


def test_special_values():
    x = torch.tensor([0.0, -0.0, 1e-42, -1e-42, 300.0, -300.0, 88.5, -88.5], device="cuda")
    gx = torch.zeros(2, 8, 384, device="cuda")
    gx[0, :, 128:256] = -200.0
    gx[0, :, 256:] = x[:, None]
    y = _run(gx)[0, :, 5]
    assert torch.equal(y[:4], x[:4]) and y[4:].tolist() == [1.0, -1.0, 1.0, -1.0]
    gx[0, :, 256:] = 50.0
    gx[1, :, 128:256] = x[:, None]
    gx[1, :, 256:] = 0.0
    y = _run(gx)[1, :, 5]
    assert y[:7].tolist() == [0.5, 0.5, 0.5, 0.5, 1.0, 0.0, 1.0] and 0.0 <= y[7].item() < 1.2e-38
    gx[1, :, 128:256] = float("nan")
    assert torch.isnan(_run(gx)[1]).all()

"""Row convolutions (`ops/conv_rows.py`, `csrc/cuda/conv_rows.cu`) against `F.conv2d` in fp64: outputs and gradients, at the
edges of the column tiles (128, 384) and chunks (32), of the groups of output rows, with remainders of the vertical stride,
even and small kernels, fewer images than blocks. TF32 operands: a few 1e-4 relative."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cin,h,w,kernel,padding", [
    (2, 1, 161, 100, (41, 11), (20, 5)),          # the speech model's first convolution
    (3, 32, 81, 50, (21, 11), (10, 5)),           # and its second
    (1, 1, 161, 771, (41, 11), (20, 5)),          # more than 384 output columns
    (1, 32, 30, 385, (21, 11), (10, 5)),
    (2, 32, 17, 128, (5, 3), (2, 1)), (1, 32, 16, 129, (4, 2), (1, 0)), (1, 32, 8, 3, (3, 3), (0, 1)), (1, 32, 1, 1, (1, 1), (0, 0)),
    (1, 32, 26, 33, (25, 16), (12, 15)), (40, 32, 11, 31, (7, 5), (3, 2)), (2, 32, 12, 257, (1, 3), (0, 1)),
    (2, 1, 33, 64, (7, 16), (2, 15)), (1, 1, 50, 65, (49, 4), (24, 0)), (1, 1, 1, 2, (1, 1), (0, 0)), (5, 1, 20, 259, (2, 3), (0, 1)),
])
def test_matches_conv2d(n, cin, h, w, kernel, padding):
    from tensorflow_allreduce_b200.ops import conv_rows, persistent_gru

    torch.manual_seed(n * 1000 + h + w)
    m = conv_rows.RowConv2d(cin, 32, kernel, stride=(2, 1 if cin == 32 else 2), padding=padding, bias=False).cuda()
    x = torch.randn(n, cin, h, w, device="cuda", requires_grad=cin == 32)
    before = conv_rows.launch_count
    y = m(x)
    wd, xd = m.weight.detach().double().requires_grad_(True), x.detach().double().requires_grad_(True)
    ref = F.conv2d(xd, wd, None, m.stride, m.padding)
    g = torch.randn_like(y)
    got = torch.autograd.grad(y, [m.weight] + ([x] if cin == 32 else []), g)
    want = torch.autograd.grad(ref, [wd, xd], g.double())
    persistent_gru.check_status()
    assert conv_rows.launch_count - before == (3 if cin == 32 else 2)
    assert y.shape == ref.shape
    for a, b in zip((y, *got), (ref, *want)):
        assert (a.double() - b).norm().item() <= 1e-3 * b.norm().item() + 1e-9


def test_other_forms_go_through_torch():
    from tensorflow_allreduce_b200.ops import conv_rows

    x = torch.randn(2, 32, 20, 30, device="cuda")
    before = conv_rows.launch_count
    for m in (conv_rows.RowConv2d(32, 32, 3, stride=1, bias=False), conv_rows.RowConv2d(32, 32, 3, stride=(2, 1)),
              conv_rows.RowConv2d(32, 16, 3, stride=(2, 1), bias=False), conv_rows.RowConv2d(32, 32, (3, 17), stride=(2, 1), bias=False)):
        m = m.cuda()
        assert torch.equal(m(x), F.conv2d(x, m.weight, m.bias, m.stride, m.padding))
    m = conv_rows.RowConv2d(32, 32, 3, stride=(2, 1), bias=False).cuda()
    old = torch.backends.cudnn.allow_tf32
    try:
        torch.backends.cudnn.allow_tf32 = False                   # fp32 asked for
        assert torch.equal(m(x), F.conv2d(x, m.weight, None, m.stride))
    finally:
        torch.backends.cudnn.allow_tf32 = old
    assert conv_rows.launch_count == before
    m(x)
    assert conv_rows.launch_count == before + 1

"""The native call paths under everything that a torch operator supports and a raw kernel does not see."""
import pytest
import torch
import torch.autograd.forward_ad as fwd
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _conv(cin=32):
    from tensorflow_allreduce_b200.ops import conv_rows

    torch.manual_seed(cin)
    m = conv_rows.RowConv2d(cin, 32, (5, 3), stride=(2, 1 if cin == 32 else 2), padding=(2, 1), bias=False).cuda()
    return m, torch.randn(2, cin, 17, 40, device="cuda", requires_grad=True)


def _stock(m, x, w):
    return F.conv2d(x, w, None, m.stride, m.padding)


def _close(got, want, rel=2e-3):
    assert (got.double() - want).norm().item() <= rel * want.norm().item() + 1e-9


@pytest.mark.parametrize("cin", [1, 32])
@pytest.mark.parametrize("strided_weight", [False, True])
def test_second_derivatives_of_a_convolution(cin, strided_weight):
    m, x = _conv(cin)
    if strided_weight:
        m.weight = torch.nn.Parameter(m.weight.detach().permute(3, 2, 1, 0).contiguous().permute(3, 2, 1, 0))
    g = torch.randn_like(m(x)).requires_grad_(True)

    def second(y, x, w, g):
        gx, gw = torch.autograd.grad(y, [x, w], g, create_graph=True)
        return [gx, gw, *torch.autograd.grad((gx ** 3).sum() + (gw ** 2).sum(), [x, w, g])]

    got = second(m(x), x, m.weight, g)
    xd, wd, gd = [t.detach().double().requires_grad_(True) for t in (x, m.weight, g)]
    for a, b in zip(got, second(_stock(m, xd, wd), xd, wd, gd)):
        _close(a, b)


def test_second_derivatives_of_the_time_first_order():
    from tensorflow_allreduce_b200 import _lib

    x = torch.randn(3, 4, 5, 70, device="cuda", requires_grad=True)
    y = _lib.ext().time_major(x)
    g = torch.randn_like(y).requires_grad_(True)
    (gx,) = torch.autograd.grad(y, x, g, create_graph=True)
    assert torch.equal(gx, g.permute(1, 2, 0).reshape(x.shape))
    v = torch.randn_like(gx)
    (gg,) = torch.autograd.grad((gx * v).sum(), g)
    assert torch.equal(gg, v.reshape(3, 20, 70).permute(2, 0, 1))


def test_second_derivative_of_the_loss_is_refused():
    from tensorflow_allreduce_b200.ops import ctc

    x = torch.randn(20, 2, 5, device="cuda", requires_grad=True)
    labels, lens = torch.randint(1, 5, (2, 4), device="cuda"), torch.tensor([4, 2], device="cuda")
    for mine in (False, True):
        logp = F.log_softmax(x, -1)
        loss = (ctc.mean_loss(logp, labels, ctc.Lengths(lens)) if mine else
                F.ctc_loss(logp, labels, torch.full((2,), 20), lens, blank=0, reduction="mean", zero_infinity=True))
        (g,) = torch.autograd.grad(loss * 3, x, create_graph=True)
        if not mine:
            first = g.detach()
        torch.testing.assert_close(g.detach(), first, rtol=1e-4, atol=1e-6)
        with pytest.raises(RuntimeError):
            torch.autograd.grad(g.square().sum(), x)


@pytest.mark.parametrize("cin", [1, 32])
def test_traced_convolution(cin):
    m, x = _conv(cin)
    with torch.no_grad():
        traced = torch.jit.trace(m, (x,))
        other = torch.randn(3, cin, 23, 50, device="cuda")
        _close(traced(other), _stock(m, other.double(), m.weight.double()))


def test_traced_time_first_order():
    from tensorflow_allreduce_b200 import _lib

    traced = torch.jit.trace(lambda x: _lib.ext().time_major(x), (torch.randn(2, 3, 5, 7, device="cuda"),), check_trace=False)
    x = torch.randn(2, 3, 5, 7, device="cuda")
    assert torch.equal(traced(x), x.reshape(2, 15, 7).permute(2, 0, 1))
    x = torch.randn(4, 6, device="cuda")
    (grad,) = torch.autograd.functional.jvp(_lib.ext().time_major, x, x)[1:]
    assert torch.equal(grad, x.t()[..., None]) and torch.equal(_lib.ext().time_major(x), x.t()[..., None])


def test_traced_loss():
    from tensorflow_allreduce_b200.ops import ctc

    labels, lens = torch.randint(1, 5, (2, 4), device="cuda"), torch.tensor([4, 2], device="cuda")

    def loss(x):
        return ctc.mean_loss(F.log_softmax(x, -1), labels, ctc.Lengths(lens))

    traced = torch.jit.trace(loss, (torch.randn(20, 2, 5, device="cuda"),), check_trace=False)
    x = torch.randn(20, 2, 5, device="cuda")
    torch.testing.assert_close(traced(x), loss(x))


@pytest.mark.parametrize("layers,nd", [(1, 1), (2, 2)])
def test_traced_gru(layers, nd):
    from tensorflow_allreduce_b200.ops import persistent_gru as pg

    class Net(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.rnn = torch.nn.GRU(40, 128, num_layers=layers, bidirectional=nd == 2)

        def forward(self, x):
            return pg.gru_forward(self.rnn, x)

    torch.manual_seed(layers)
    net = Net().cuda().eval()
    traced = torch.jit.trace(net, (torch.randn(6, 3, 40, device="cuda"),), check_trace=False)
    x = torch.randn(9, 2, 40, device="cuda", requires_grad=True)
    want = net(x)
    before = pg.launch_count
    y = traced(x)
    assert pg.launch_count == before
    _close(y, want.double())
    for a, b in zip(torch.autograd.grad(y.sum(), [x, *net.parameters()]), torch.autograd.grad(want.sum(), [x, *net.parameters()])):
        _close(a, b.double(), 5e-3)


def test_traced_norm():
    from tensorflow_allreduce_b200.ops import bn_clip

    class Net(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.a, self.b = bn_clip.BatchNormClip2d(4), bn_clip.BatchNormClip2d(4, clip=1.0)

        def forward(self, x):
            return self.a(x), bn_clip.bn_clip(x, self.b.weight, self.b.bias, None, None, 1e-5, 0.1, 1.0)

    net = Net().cuda()
    traced = torch.jit.trace(net, (torch.randn(3, 4, 5, 6, device="cuda"),), check_trace=False)
    x = torch.randn(2, 4, 7, 6, device="cuda")
    count = net.a.num_batches_tracked.item()
    for a, b in zip(traced(x), net(x)):
        torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-5)
    assert net.a.num_batches_tracked.item() == count + 2


@pytest.mark.parametrize("cin", [1, 32])
def test_forward_mode_through_a_convolution(cin):
    m, x = _conv(cin)
    t = torch.randn_like(x)
    with fwd.dual_level():
        y = fwd.unpack_dual(m(fwd.make_dual(x.detach(), t)))
    _close(y.primal, _stock(m, x.detach().double(), m.weight.double()))
    _close(y.tangent, _stock(m, t.double(), m.weight.double()))


def test_forward_mode_through_the_time_first_order():
    from tensorflow_allreduce_b200 import _lib

    x, t = torch.randn(2, 3, 5, 7, device="cuda"), torch.randn(2, 3, 5, 7, device="cuda")
    with fwd.dual_level():
        y = fwd.unpack_dual(_lib.ext().time_major(fwd.make_dual(x, t)))
    assert torch.equal(y.tangent, t.reshape(2, 15, 7).permute(2, 0, 1))


def test_forward_mode_through_a_gru_is_refused():
    from tensorflow_allreduce_b200.ops import persistent_gru as pg

    rnn = torch.nn.GRU(40, 128).cuda()
    x = torch.randn(6, 3, 40, device="cuda")
    for p in rnn.parameters():
        p.requires_grad_(False)
    with fwd.dual_level():
        with pytest.raises(RuntimeError):
            pg.gru_forward(rnn, fwd.make_dual(x, torch.ones_like(x)))


def test_forward_mode_through_a_norm_is_refused():
    from tensorflow_allreduce_b200.ops import bn_clip

    m = bn_clip.BatchNormClip2d(4).cuda()
    x = torch.randn(3, 4, 5, 6, device="cuda")
    with fwd.dual_level():
        with pytest.raises(RuntimeError):
            m(fwd.make_dual(x, torch.ones_like(x)))


@pytest.mark.parametrize("cin", [1, 32])
def test_batches_of_gradients_and_vmap(cin):
    m, x = _conv(cin)
    y = m(x)
    g = torch.randn(3, *y.shape, device="cuda")
    gx, gw = torch.autograd.grad(y, [x, m.weight], g, is_grads_batched=True)
    for i in range(3):
        xd, wd = x.detach().double().requires_grad_(True), m.weight.detach().double().requires_grad_(True)
        wx, ww = torch.autograd.grad(_stock(m, xd, wd), [xd, wd], g[i].double())
        _close(gx[i], wx)
        _close(gw[i], ww)
    xs = torch.randn(3, *x.shape, device="cuda")
    with torch.no_grad():
        _close(torch.vmap(m)(xs), torch.stack([_stock(m, v.double(), m.weight.double()) for v in xs]))
    f = torch.func.grad(lambda w: torch.func.functional_call(m, {"weight": w}, (x.detach(),)).square().sum())
    wd = m.weight.detach().double().requires_grad_(True)
    _close(f(m.weight.detach()), torch.autograd.grad(_stock(m, x.detach().double(), wd).square().sum(), wd)[0])


def test_batches_of_gradients_of_the_time_first_order_and_the_loss():
    from tensorflow_allreduce_b200 import _lib
    from tensorflow_allreduce_b200.ops import ctc

    x = torch.randn(2, 3, 5, 7, device="cuda", requires_grad=True)
    y = _lib.ext().time_major(x)
    g = torch.randn(4, *y.shape, device="cuda")
    (gx,) = torch.autograd.grad(y, x, g, is_grads_batched=True)
    assert torch.equal(gx, torch.stack([v.permute(1, 2, 0).reshape(x.shape) for v in g]))
    with torch.no_grad():
        xs = torch.randn(4, 2, 3, 5, 7, device="cuda")
        assert torch.equal(torch.vmap(lambda v: _lib.ext().time_major(v))(xs), torch.stack([v.reshape(2, 15, 7).permute(2, 0, 1) for v in xs]))
    s = torch.randn(20, 2, 5, device="cuda", requires_grad=True)
    labels, lens = torch.randint(1, 5, (2, 4), device="cuda"), torch.tensor([4, 2], device="cuda")
    loss = ctc.mean_loss(F.log_softmax(s, -1), labels, ctc.Lengths(lens))
    (one,) = torch.autograd.grad(loss, s, retain_graph=True)
    (many,) = torch.autograd.grad(loss, s, torch.tensor([1.0, -2.0], device="cuda"), is_grads_batched=True)
    torch.testing.assert_close(many, torch.stack([one, -2 * one]))


def test_dispatch_modes_see_the_operators():
    from torch.utils.flop_counter import FlopCounterMode

    m, x = _conv()
    with FlopCounterMode(display=False) as mine, torch.no_grad():
        m(x)
    with FlopCounterMode(display=False) as stock, torch.no_grad():
        _stock(m, x, m.weight)
    assert mine.get_total_flops() == stock.get_total_flops() > 0


def test_precision_asked_for_by_operator():
    m, x = _conv()
    before = torch.backends.cudnn.conv.fp32_precision
    want = _stock(m, x.double(), m.weight.double())
    try:
        torch.backends.cudnn.conv.fp32_precision = "ieee"
        _close(m(x), want, 1e-5)
    finally:
        torch.backends.cudnn.conv.fp32_precision = before
    with torch.backends.cudnn.flags(enabled=False):
        _close(m(x), want, 1e-5)


def test_norm_whose_buffers_lie_elsewhere():
    from tensorflow_allreduce_b200.ops import bn_clip

    torch.manual_seed(0)
    x = torch.randn(3, 4, 5, 6, device="cuda")
    want = bn_clip.BatchNormClip2d(4).cuda()
    y = want(x)
    for count in (torch.tensor(7), torch.tensor(7, device="cuda", dtype=torch.int32), torch.tensor(7, device="cuda"), None):
        m = bn_clip.BatchNormClip2d(4).cuda()
        m.num_batches_tracked = count
        before = bn_clip.launch_count
        assert torch.equal(m(x), y) and bn_clip.launch_count == before + 1
        assert count is None or (m.num_batches_tracked.item() == 8 and m.num_batches_tracked.device == count.device)
        assert torch.equal(m.running_mean, want.running_mean) and torch.equal(m.running_var, want.running_var)
    m = bn_clip.BatchNormClip2d(4).cuda()
    both = torch.zeros(4, 2, device="cuda")
    m.running_mean = both[:, 0]
    m.weight = torch.nn.Parameter(torch.ones(4, 3, device="cuda")[:, 1])
    torch.testing.assert_close(m(x), y, rtol=1e-5, atol=1e-5)
    assert (both[:, 1] == 0).all() and m.num_batches_tracked.item() == 1
    m = bn_clip.BatchNormClip2d(4).cuda()
    m.running_mean = torch.zeros(4)
    with pytest.raises(RuntimeError):
        m(x)

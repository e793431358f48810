"""What the blocks of a persistent GRU layer exchange: factors formed by the forward pass against factors formed in the backward pass,
values that are not finite, pairs of blocks under a CUDA graph."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,B", [(128, 1), (128, 17), (256, 16), (384, 32), (640, 5), (896, 31), (1024, 32)])
def test_factors_of_either_pass(H, B):
    # The same function of the same fp32 values, so the same bits.
    from tensorflow_allreduce_b200 import _lib

    lib, T, nd = _lib.lib(), 5, 2
    torch.manual_seed(H + B)
    f = lambda *s: torch.randn(*s, device="cuda")
    w, b = [f(3 * H, H) / H ** 0.5 for _ in range(2)], [f(3 * H) for _ in range(2)]
    gx, dy = f(T, B, nd, 3 * H), f(T, B, nd * H)
    scratch = torch.zeros(lib.bc_gru_scratch_bytes(T, B, H, nd), dtype=torch.uint8, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    got = []
    for factors in (False, True):
        y, dg, db = f(T, B, nd * H), f(T * B, nd * 4 * H), f(nd, 2, 3 * H)
        if factors:
            keep = f(nd, T, B, 5, H)
            _lib.check(lib.bc_gru_forward_factors(T, B, H, nd, *map(p, w + b), p(gx), p(y), p(keep), p(scratch), p(status), 10.0, stream), "forward")
            _lib.check(lib.bc_gru_backward_factors(T, B, H, nd, *map(p, w), p(keep), p(dy), p(dg), p(db), p(scratch), p(status), 10.0, stream), "backward")
        else:
            keep = f(nd, T, B, H, 4)
            _lib.check(lib.bc_gru_forward(T, B, H, nd, *map(p, w + b), p(gx), p(y), p(keep), p(scratch), p(status), 10.0, stream), "forward")
            _lib.check(lib.bc_gru_backward(T, B, H, nd, *map(p, w), p(y), p(keep), p(dy), p(dg), p(db), p(scratch), p(status), 10.0, stream), "backward")
        got.append((y, dg, db))
    assert status.item() == 0
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("H,B", [(128, 3), (512, 17), (1024, 32)])
def test_nan_stays_in_its_batch_entry(H, B):
    from tensorflow_allreduce_b200.ops import persistent_gru as pg

    torch.manual_seed(H)
    rnn, x = torch.nn.GRU(24, H).cuda(), torch.randn(6, B, 24, device="cuda")
    bad = x.clone()
    bad[2, B - 1] = float("nan")
    out = []
    for v in (x, bad):
        v.requires_grad_(True)
        y = pg.gru_forward(rnn, v)
        out.append((y.detach(), *torch.autograd.grad(y, v, torch.ones_like(y))))
    pg.check_status()
    (y0, d0), (y1, d1) = out
    assert torch.equal(y0[:2], y1[:2]) and torch.equal(y0[:, :B - 1], y1[:, :B - 1]) and torch.isnan(y1[2:, B - 1]).all()
    assert torch.equal(d0[:, :B - 1], d1[:, :B - 1]) and torch.isnan(d1[:, B - 1]).all()


def test_large_and_infinite_weights():
    # fp16 has no 1e6: the rows are scaled. An infinite weight is one, not a NaN, where h is not zero.
    from tensorflow_allreduce_b200.ops import persistent_gru as pg

    torch.manual_seed(0)
    rnn, x = torch.nn.GRU(24, 128).cuda(), torch.randn(4, 3, 24, device="cuda")
    with torch.no_grad():
        rnn.weight_hh_l0[:64] *= 1e6
        rnn.weight_hh_l0[64:128] *= 1e-9
        want = torch.nn.GRU(24, 128).cuda().double()
        want.load_state_dict(rnn.state_dict())
        with torch.backends.cudnn.flags(enabled=False):
            ref = want(x.double())[0]
        y = pg.gru_forward(rnn, x)
        assert (y - ref).norm() <= 2e-3 * ref.norm()          # saturated gates; the rest as in test_gpu_persistent_gru_sizes.py
        rnn.weight_hh_l0[130, 5] = float("inf")               # update gate of unit 2
        y = pg.gru_forward(rnn, x)
    pg.check_status()
    assert torch.isfinite(y).all()


def test_pairs_of_blocks_in_a_graph():
    from tensorflow_allreduce_b200.ops import persistent_gru as pg

    torch.manual_seed(1)
    rnn, x = torch.nn.GRU(24, 512, bidirectional=True).cuda(), torch.randn(8, 20, 24, device="cuda")
    with torch.no_grad():
        want = pg.gru_forward(rnn, x)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y = pg.gru_forward(rnn, x)
        graph.replay()
        graph.replay()
    torch.cuda.synchronize()
    pg.check_status()
    assert torch.equal(y, want)


def test_saved_tensors_that_come_back_as_views(monkeypatch):
    # A hook may put what it is given anywhere: here 16 bytes behind a multiple of 32, which the recurrent weights are read at.
    from tensorflow_allreduce_b200.ops import persistent_gru as pg

    def pack(t):
        room = torch.empty(t.numel() + 4, device=t.device, dtype=t.dtype)
        return room[4:].copy_(t.detach().reshape(-1)).view(t.shape)

    monkeypatch.setattr(torch.backends.cuda.matmul, "allow_tf32", False)      # whatever GEMM an alignment selects
    torch.manual_seed(2)
    rnn, x = torch.nn.GRU(24, 256, bidirectional=True).cuda(), torch.randn(6, 5, 24, device="cuda", requires_grad=True)
    params = [x, *rnn.parameters()]
    y = pg.gru_forward(rnn, x)
    want = torch.autograd.grad(y, params, torch.ones_like(y))
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        y = pg.gru_forward(rnn, x)
    got = torch.autograd.grad(y, params, torch.ones_like(y))
    pg.check_status()
    for a, b in zip(got, want):
        assert (a - b).norm() <= 1e-5 * b.norm()          # library GEMMs may take another path at another alignment

"""Bounded waits of the persistent GRU kernels and the row convolutions that run out. GRU: the meeting of a direction's blocks is given a counter that never fills, or the
words that the blocks exchange are wiped while they are on their way. The kernels end by themselves and say so in the status word; the next
call is right. The limit is two milliseconds. Convolutions: inputs that lie in pinned host memory, which take longer to load than the limit of a
microsecond allows the tensor cores to wait for them."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

LIMIT = 2e-3


class Layer:
    """A layer's tensors, called through the C entry points with memory and a status word of the caller's."""

    def __init__(self, H, B, T, seed=0):
        from tensorflow_allreduce_b200 import _lib

        self._lib = _lib
        self.lib = _lib.lib()
        self.T, self.B, self.H = T, B, H
        torch.manual_seed(seed)
        f = lambda *s: torch.randn(*s, device="cuda")
        self.w, self.b = [f(3 * H, H) / H ** 0.5 for _ in range(2)], [f(3 * H) for _ in range(2)]
        self.gx, self.y, self.rsv, self.dy = f(T, B, 2, 3 * H), f(T, B, 2 * H), f(2, T, B, H, 4), f(T, B, 2 * H)
        self.dg, self.db = f(T * B, 8 * H), f(2, 2, 3 * H)
        self.status = torch.zeros(1, dtype=torch.int32, device="cuda")
        self.other = torch.cuda.Stream()

    def run(self, backward, arrivals=0, wipes=0):
        """`arrivals`: what the counter of direction 0 starts from; `wipes`: how often the words are wiped meanwhile, from another stream.
        Returns status and outputs."""
        p = lambda t: C.c_void_p(t.data_ptr())
        scratch = torch.zeros(self.lib.bc_gru_scratch_bytes(self.T, self.B, self.H, 2), dtype=torch.uint8, device="cuda")
        scratch[:4].view(torch.int32).fill_(arrivals)
        self.status.zero_()
        torch.cuda.synchronize()
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        if backward:
            rc = self.lib.bc_gru_backward(self.T, self.B, self.H, 2, p(self.w[0]), p(self.w[1]), p(self.y), p(self.rsv), p(self.dy), p(self.dg), p(self.db),
                                          p(scratch), p(self.status), LIMIT, stream)
            out = [self.dg, self.db]
        else:
            rc = self.lib.bc_gru_forward(self.T, self.B, self.H, 2, p(self.w[0]), p(self.w[1]), p(self.b[0]), p(self.b[1]), p(self.gx), p(self.y), p(self.rsv),
                                         p(scratch), p(self.status), LIMIT, stream)
            out = [self.y, self.rsv]
        self._lib.check(rc, "GRU pass")
        with torch.cuda.stream(self.other):
            for _ in range(wipes):
                scratch[1024:].zero_()
        torch.cuda.synchronize()
        return self.status.item(), [t.clone() for t in out]


SHAPES = [(128, 4, 9), (512, 8, 20), (1024, 32, 40)]


@pytest.mark.parametrize("backward", [False, True])
@pytest.mark.parametrize("H,B,T", SHAPES)
def test_blocks_that_never_meet(H, B, T, backward):
    l = Layer(H, B, T)
    if backward:
        l.run(False)
    code, want = l.run(backward)
    assert code == 0
    assert l.run(backward, arrivals=1 << 20)[0] != 0
    code, got = l.run(backward)
    assert code == 0 and all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("backward", [False, True])
@pytest.mark.parametrize("H,B", [(128, 4), (512, 8), (1024, 32)])
def test_words_that_do_not_arrive(H, B, backward):
    # A word that is wiped before it is read is waited for until the limit, one that is wiped later does no harm: a launch that reports nothing is
    # right. A launch of 700 steps lasts about a millisecond, some hundred wipes.
    l = Layer(H, B, 700)
    if backward:
        l.run(False)
    code, want = l.run(backward)
    assert code == 0
    codes = []
    for _ in range(5):
        code, got = l.run(backward, wipes=200)
        codes.append(code)
        assert code != 0 or all(torch.equal(a, b) for a, b in zip(got, want))
    print(codes)
    assert any(codes)
    code, got = l.run(backward)
    assert code == 0 and all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("cin", [1, 32])
@pytest.mark.parametrize("which", ["forward", "input", "weight"])
def test_convolution_whose_input_comes_late(which, cin):
    from tensorflow_allreduce_b200 import _lib

    if which == "input" and cin == 1:
        pytest.skip("the gradient of a single input channel is torch's")
    lib = _lib.lib()
    n, h, w, k = 16, 81, 350, (21, 11)
    sw = 1 if cin == 32 else 2
    ho, wo = (h + 20 - 21) // 2 + 1, (w + 10 - 11) // sw + 1
    dims = (C.c_int * 9)(n, cin, h, w, *k, 10, 5, sw)
    torch.manual_seed(0)
    x, dy = torch.randn(n, cin, h, w, device="cuda"), torch.randn(n, 32, ho, wo, device="cuda")
    weight = torch.randn(32, cin, *k, device="cuda")
    scratch = torch.empty(lib.bc_conv_scratch_bytes(dims), dtype=torch.uint8, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def run(x, dy, limit):
        out = torch.zeros_like({"forward": dy, "input": x, "weight": weight}[which], device="cuda")
        if which == "forward":
            rc = lib.bc_conv_forward(dims, p(x), p(weight), p(out), p(scratch), p(status), C.c_double(limit), stream)
        elif which == "input":
            rc = lib.bc_conv_backward_input(dims, p(dy), p(weight), p(out), p(scratch), p(status), C.c_double(limit), stream)
        else:
            rc = lib.bc_conv_backward_weight(dims, p(x), p(dy), p(out), p(scratch), p(status), C.c_double(limit), stream)
        _lib.check(rc, which)
        code = status.item()
        status.zero_()
        return code, out

    code, want = run(x, dy, 10.0)
    assert code == 0
    late = x.cpu().pin_memory(), dy.cpu().pin_memory()
    code, got = run(*late, 10.0)                       # late, but in time
    assert code == 0 and torch.equal(got, want)
    assert run(*late, 1e-6)[0] == 8
    code, got = run(x, dy, 10.0)
    assert code == 0 and torch.equal(got, want)

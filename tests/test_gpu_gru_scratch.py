"""The memory through which the blocks of a persistent GRU layer exchange: under CUDA graphs, with several threads on a stream, with many
streams."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(H, B=5, T=12, seed=0):
    torch.manual_seed(seed)
    return torch.nn.GRU(24, H, bidirectional=True).cuda(), torch.randn(T, B, 24, device="cuda", requires_grad=True)


def _pass(rnn, x):
    from tensorflow_allreduce_b200.ops import persistent_gru as pg

    y = pg.gru_forward(rnn, x)
    return [y.detach(), *torch.autograd.grad(y, [x, *rnn.parameters()], torch.ones_like(y))]


def test_graphs_in_any_order_and_at_a_time():
    from tensorflow_allreduce_b200.ops import persistent_gru as pg

    layers = [_layer(128, seed=1), _layer(256, seed=2)]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        want = [[t.clone() for t in _pass(*l)] for l in layers]
    torch.cuda.current_stream().wait_stream(side)
    graphs, outs = [], []
    for l in layers:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            outs.append(_pass(*l))
        graphs.append(g)

    def check(i):
        torch.cuda.synchronize()
        pg.check_status()
        for a, b in zip(outs[i], want[i]):
            assert torch.equal(a, b)
            a.zero_()

    graphs[1].replay()
    check(1)
    graphs[0].replay()
    check(0)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(50):
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
    check(0)
    check(1)
    del graphs[0]
    with torch.cuda.stream(side):
        got = _pass(*layers[0])
    torch.cuda.synchronize()
    for a, b in zip(got, want[0]):
        assert torch.equal(a, b)


def test_threads_on_one_stream():
    from tensorflow_allreduce_b200.ops import persistent_gru as pg

    sizes = [(128, 2), (256, 9), (384, 17), (512, 32)]
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        layers = [_layer(h, b, 7, seed=h) for h, b in sizes]
        want = [_pass(*l) for l in layers]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        with torch.cuda.stream(stream):
            for _ in range(10):
                for j in range(len(layers)):
                    k = (i + j) % len(layers)
                    got = _pass(*layers[k])
                    if not all(torch.equal(a, b) for a, b in zip(got, want[k])):
                        wrong.append(k)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    pg.check_status()
    assert not wrong


def test_many_streams_do_not_hold_more_and_more_memory():
    from tensorflow_allreduce_b200 import _lib

    from tensorflow_allreduce_b200.ops import persistent_gru as pg

    rnn, x = _layer(1024, 32, 2)
    size = _lib.lib().bc_gru_scratch_bytes(2, 32, 1024, 2)
    streams = [torch.cuda.Stream() for _ in range(24)] + [torch.cuda.Stream(priority=-1) for _ in range(24)]
    assert len({s.cuda_stream for s in streams}) > 32
    held = []
    with torch.no_grad():
        for rounds in range(2):
            for s in streams:
                with torch.cuda.stream(s):
                    torch.mm(x[0], x[0].t())               # torch keeps a workspace for the products of each stream
                    if rounds:
                        pg.gru_forward(rnn, x)
            torch.cuda.synchronize()
            held.append(torch.cuda.memory_allocated())
    assert held[1] - held[0] <= 17 * size


def test_status_is_that_of_all_streams():
    from tensorflow_allreduce_b200.ops import persistent_gru as pg

    rnn, x = _layer(128)
    _pass(rnn, x)
    side, done = torch.cuda.Stream(), torch.cuda.Event()
    with torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)                # about a tenth of a second
        _pass(rnn, x)
        done.record()
    pg.check_status()
    assert done.query()


def test_status_word_of_a_first_call_that_is_captured():
    # In a process of its own: the status word is made by the first call. Memory of the graphs' pool that held other values before must not pass
    # for it.
    import os
    import subprocess
    import sys

    code = """
import torch
from tensorflow_allreduce_b200.ops import persistent_gru as pg
rnn, x = torch.nn.GRU(24, 128).cuda(), torch.randn(7, 5, 24, device="cuda")
with torch.no_grad():
    want = rnn(x)[0]
    torch.addmm(rnn.bias_ih_l0, x[0], rnn.weight_ih_l0.t())
    torch.cuda.synchronize()
    first, second = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(first):
        junk = [torch.full((60000,), 7, dtype=torch.int32, device="cuda") for _ in range(8)]
        del junk
    first.replay()
    with torch.cuda.graph(second, pool=first.pool()):
        y = pg.gru_forward(rnn, x)
    pg.check_status()
    second.replay()
    pg.check_status()
    assert (y - want).abs().max().item() < 5e-3
print("right")
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=120)
    assert res.returncode == 0 and "right" in res.stdout, res.stdout + res.stderr

"""CTC loss (`ops/ctc.py`, `csrc/cuda/ctc.cu`) against `F.ctc_loss` in fp64 on the CPU: loss and gradient with respect to the scores
in front of the softmax. One frame, one state, states that fill warps and the block, frames that do not divide by the steps in flight
or the frames per block, repeated labels, utterances without a path, empty ones."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,b,c,longest", [
    (350, 32, 29, 100), (1, 1, 2, 0), (1, 2, 5, 1), (7, 3, 3, 4), (8, 3, 29, 3), (9, 2, 40, 15), (16, 5, 29, 16), (17, 2, 200, 8), (63, 4, 2, 31),
    (64, 1, 29, 32), (100, 2, 29, 99), (1100, 2, 29, 511), (33, 70, 6, 12),
])
def test_matches_ctc_loss(t, b, c, longest):
    from tensorflow_allreduce_b200.ops import ctc

    torch.manual_seed(t * 1000 + longest)
    x = torch.randn(t, b, c, device="cuda", requires_grad=True)
    labels = torch.randint(1, max(c, 2), (b, longest), device="cuda")
    lens = torch.randint(0, longest + 1, (b,), device="cuda")
    lens[0] = longest
    before = ctc.launch_count
    loss = ctc.mean_loss(F.log_softmax(x, -1), labels, ctc.Lengths(lens))
    (grad,) = torch.autograd.grad(loss * 3, x)
    assert ctc.launch_count == before + 2
    xd = x.detach().double().cpu().requires_grad_(True)
    want = F.ctc_loss(F.log_softmax(xd, -1), labels.cpu(), torch.full((b,), t), lens.cpu(), blank=0, reduction="mean", zero_infinity=True)
    (wgrad,) = torch.autograd.grad(want * 3, xd)
    assert abs(loss.item() - want.item()) <= 1e-5 * abs(want.item()) + 1e-6
    # Sums of t logarithms in fp32 round the more, the longer they are: torch's own fp32 gradient is the measure.
    xt = x.detach().requires_grad_(True)
    theirs = F.ctc_loss(F.log_softmax(xt, -1), labels, torch.full((b,), t), lens, blank=0, reduction="mean", zero_infinity=True)
    (tgrad,) = torch.autograd.grad(theirs * 3, xt)
    mine, torchs = [(g.cpu().double() - wgrad).norm().item() / (wgrad.norm().item() + 1e-9) for g in (grad, tgrad)]
    print(f"relative error {mine:.2e}, torch {torchs:.2e}")
    assert mine <= 1.2 * torchs + 5e-6


def test_wrong_lengths_are_refused():
    from tensorflow_allreduce_b200.ops import ctc

    logp = F.log_softmax(torch.randn(10, 2, 5, device="cuda"), -1)
    labels = torch.ones(2, 3, dtype=torch.int64, device="cuda")
    for bad in ([3, 4], [-1, 2]):
        with pytest.raises(RuntimeError):
            ctc.mean_loss(logp, labels, ctc.Lengths(torch.tensor(bad, device="cuda")))
    assert ctc.mean_loss(logp.double(), labels, ctc.Lengths(torch.tensor([3, 2], device="cuda"))).dtype == torch.float64

"""CTC loss of batches whose utterances all have as many frames, on the library's kernels (`csrc/cuda/ctc.cu`).

`mean_loss` is `F.ctc_loss(..., blank=0, reduction="mean", zero_infinity=True)` with input lengths of T. On fp32 CUDA
log-probabilities with [batch, length] int64 labels of up to 511 it is three kernels, forward and backward, without a wait for
the device in between; everything else is `F.ctc_loss`, which copies the lengths in both directions and waits for each copy.

The reference computes the loss on the CPU (tensorflow/core/kernels/ctc_loss_op.cc:167).
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

from .. import _lib


def __getattr__(name):
    if name == "launch_count":   # passes (forward, backward) run by this process
        return int(_lib.ext().ctc_launches())
    raise AttributeError(name)


class Lengths:
    """Label lengths on their way to the host, which has to know them to reject wrong ones. Made before a forward pass is
    queued and read after it, the copy is over by the time that the device has caught up, and the host does not wait for the pass."""

    def __init__(self, lengths: torch.Tensor):
        self.device = lengths
        self.event = None
        self.host = lengths
        if lengths.is_cuda and _lib.ext().plain(lengths):
            with torch.cuda.device(lengths.device):
                self.host = torch.empty(lengths.shape, dtype=lengths.dtype, pin_memory=True)
                self.host.copy_(lengths, non_blocking=True)
                self.event = torch.cuda.Event()
                self.event.record()

    def check(self, longest: int) -> None:
        if self.event is not None:
            self.event.synchronize()
        for n in self.host.tolist():
            if not 0 <= n <= longest:
                raise RuntimeError(f"label length {n} is outside the labels given, 0 to {longest}")


def mean_loss(logp: torch.Tensor, labels: torch.Tensor, lengths: Lengths) -> torch.Tensor:
    """logp: [T, B, C] log-probabilities out of a softmax; labels: [B, L]; class 0 is the blank."""
    t, b, _ = logp.shape
    n = lengths.device
    if (logp.is_cuda and _lib.ext().plain(logp) and logp.dtype == torch.float32 and logp.numel() > 0 and labels.dim() == 2 and labels.dtype == torch.int64
            and labels.device == logp.device and labels.shape[0] == b <= 65535 and labels.shape[1] <= 511
            and n.dtype == torch.int64 and tuple(n.shape) == (b,)
            and _lib.ext().plain(labels) and _lib.ext().plain(n)):
        lengths.check(labels.shape[1])
        return _lib.ext().ctc_mean(logp, labels, n.to(logp.device, non_blocking=True))
    in_len = torch.full((b,), t, dtype=torch.long, device=logp.device)
    return F.ctc_loss(logp, labels, in_len, n, blank=0, reduction="mean", zero_infinity=True)

"""Persistent GRU layers on the tcgen05 kernels of `csrc/cuda/gru_forward.cu` and `gru_backward.cu`.

A GRU layer is split the usual way into the input projections of all time steps (one library
GEMM) and the recurrence. The recurrence of both directions of a layer runs in ONE cooperative
kernel launch whose blocks keep their slice of the recurrent weights on chip for the whole
sequence; see the kernel file for the design (the call path around it is native, `csrc/torch/bindings.cc`). The reference's counterparts launch at least
one GEMM and one elementwise kernel per time step (tensorflow/contrib/rnn/kernels/gru_ops.h:69-119,
contrib/cudnn_rnn/kernels/cudnn_rnn_ops.cc:738-1091).

`gru_forward(rnn, x)` evaluates a `torch.nn.GRU` with its own parameters (same gate order and
equations as `torch.nn.GRU`, zero initial state, time-major input) and is differentiable, so a
model keeps its `nn.GRU` module, parameters and `state_dict` and only swaps the call.
"""
from __future__ import annotations

import os
from typing import List

import torch

from .. import _lib

_TIMEOUT_S = float(os.environ.get("BC_GRU_TIMEOUT_S", "10"))   # bound of every wait inside the kernels


def __getattr__(name):
    if name == "launch_count":   # persistent kernels launched by this process (forward and backward)
        return int(_lib.ext().gru_launches())
    raise AttributeError(name)


def _ext():
    e = _lib.ext()
    if not getattr(e, "_gru_ready", False):
        e.gru_set_timeout(_TIMEOUT_S)
        e._gru_ready = True
    return e


def check_status(device=None) -> None:
    """Raise if a persistent GRU kernel on `device` gave up on a bounded wait since the last
    check (this synchronises with the device)."""
    e = _lib.ext()
    for idx in e.gru_devices():
        if device is not None and torch.device(device).index not in (None, idx):
            continue
        code = e.gru_take_status(idx)
        if code:
            if code & 8:
                raise RuntimeError(f"a row convolution timed out on cuda:{idx} (status 0x{code:x}); its outputs are incomplete")
            raise RuntimeError(f"a persistent GRU kernel timed out on cuda:{idx} (status 0x{code:x}); its outputs are incomplete")


def supported(T: int, B: int, H: int, ndir: int, device=None) -> bool:
    """Can the persistent kernels run these dimensions on this device? (B <= 32, H a multiple of
    128 up to 1024, a compute-capability-10 GPU with enough SMs for H/16 blocks per direction.)"""
    if not torch.cuda.is_available():
        return False
    dev = torch.device(device) if device is not None else torch.device("cuda", torch.cuda.current_device())
    idx = dev.index if dev.index is not None else torch.cuda.current_device()
    return _lib.lib().bc_gru_supported(idx, int(T), int(B), int(H), int(ndir)) == 1


def _stack(x: torch.Tensor, weights: List[torch.Tensor], layers: int) -> torch.Tensor:
    if torch._C._get_tracing_state() is not None:      # a trace does not see the kernels: it holds torch's operator
        nd = len(weights) // (4 * layers)
        h = torch.zeros(layers * nd, x.shape[1], weights[1].shape[1], device=x.device)
        return torch._VF.gru(x, h, weights, True, layers, 0.0, True, nd == 2, False)[0]
    return _ext().gru_stack(x, weights, layers)


def gru_layer(x: torch.Tensor, w_ih: torch.Tensor, w_hh: torch.Tensor, b_ih: torch.Tensor, b_hh: torch.Tensor) -> torch.Tensor:
    """One GRU layer over a time-major fp32 sequence x [T, B, I] with zero initial state.
    Parameters are stacked over the directions (1 or 2). Returns [T, B, ndir * H]."""
    return _stack(x, [t[d] for d in range(w_hh.shape[0]) for t in (w_ih, w_hh, b_ih, b_hh)], 1)


def gru_forward(rnn: torch.nn.GRU, x: torch.Tensor) -> torch.Tensor:
    """`rnn(x)[0]` for a time-major `torch.nn.GRU` with biases and zero initial state, computed by
    the persistent kernels. Raises if the module or the shapes are not supported (use `supported`)."""
    if rnn.batch_first or not rnn.bias or rnn.dropout != 0.0 or getattr(rnn, "proj_size", 0):
        raise ValueError("gru_forward needs a time-major nn.GRU with biases, no dropout and no projection")
    nd = 2 if rnn.bidirectional else 1
    weights: List[torch.Tensor] = []
    for layer in range(rnn.num_layers):
        for sfx in (f"_l{layer}", f"_l{layer}_reverse")[:nd]:
            weights += (getattr(rnn, "weight_ih" + sfx), getattr(rnn, "weight_hh" + sfx), getattr(rnn, "bias_ih" + sfx), getattr(rnn, "bias_hh" + sfx))
    return _stack(x, weights, rnn.num_layers)

"""Persistent GRU layers on the tcgen05 kernels of `csrc/cuda/gru_persistent.cu`.

A GRU layer is split the usual way into the input projections of all time steps (one library
GEMM) and the recurrence. The recurrence of both directions of a layer runs in ONE cooperative
kernel launch whose blocks keep their slice of the recurrent weights on chip for the whole
sequence; see the kernel file for the design. The reference's counterparts launch at least
one GEMM and one elementwise kernel per time step (tensorflow/contrib/rnn/kernels/gru_ops.h:69-119,
contrib/cudnn_rnn/kernels/cudnn_rnn_ops.cc:738-1091).

`gru_forward(rnn, x)` evaluates a `torch.nn.GRU` with its own parameters (same gate order and
equations as `torch.nn.GRU`, zero initial state, time-major input) and is differentiable, so a
model keeps its `nn.GRU` module, parameters and `state_dict` and only swaps the call.
"""
from __future__ import annotations

import ctypes as C
import os
from typing import Dict, List, Optional, Tuple

import torch

from .. import _lib

_TIMEOUT_S = float(os.environ.get("BC_GRU_TIMEOUT_S", "10"))   # bound of every wait inside the kernels
_status: Dict[int, torch.Tensor] = {}
launch_count = 0   # persistent kernels launched by this process (forward and backward)


def _status_word(device: torch.device) -> torch.Tensor:
    idx = device.index if device.index is not None else torch.cuda.current_device()
    t = _status.get(idx)
    if t is None:
        t = torch.zeros(1, dtype=torch.int32, device=device)
        _status[idx] = t
    return t


_scratch_of: Dict[Tuple[int, int], torch.Tensor] = {}


def _scratch(device: torch.device, stream: int, T: int, B: int, H: int, nd: int) -> torch.Tensor:
    """Memory through which the blocks of a launch exchange operands and partial sums. Every word says which
    step it belongs to and a launch clears its part first, so the contents only have to be zero once.
    Kernels on one stream use it one after the other: one buffer per device and stream."""
    key = (device.index if device.index is not None else torch.cuda.current_device(), stream)
    need = int(_lib.lib().bc_gru_scratch_bytes(T, B, H, nd))
    t = _scratch_of.get(key)
    if t is None or t.numel() < need:
        t = torch.zeros(need, dtype=torch.uint8, device=device)
        _scratch_of[key] = t
    return t


def check_status(device=None) -> None:
    """Raise if a persistent GRU kernel on `device` gave up on a bounded wait since the last
    check (this synchronises with the device)."""
    for idx, t in list(_status.items()):
        if device is not None and torch.device(device).index not in (None, idx):
            continue
        code = int(t.item())
        if code:
            t.zero_()
            for key, w in _scratch_of.items():
                if key[0] == idx:
                    w.zero_()
            raise RuntimeError(f"a persistent GRU kernel timed out on cuda:{idx} (status 0x{code:x}); its outputs are incomplete")


def supported(T: int, B: int, H: int, ndir: int, device=None) -> bool:
    """Can the persistent kernels run these dimensions on this device? (B <= 32, H a multiple of
    128 up to 1024, a compute-capability-10 GPU with enough SMs for H/16 blocks per direction.)"""
    if not torch.cuda.is_available():
        return False
    dev = torch.device(device) if device is not None else torch.device("cuda", torch.cuda.current_device())
    idx = dev.index if dev.index is not None else torch.cuda.current_device()
    return _lib.lib().bc_gru_supported(idx, int(T), int(B), int(H), int(ndir)) == 1


def _ptr(t: Optional[torch.Tensor]):
    return C.c_void_p(t.data_ptr()) if t is not None else None


def _aligned(t: torch.Tensor) -> torch.Tensor:
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _forward(x: torch.Tensor, weights: List[torch.Tensor], save: bool):
    """Output of one layer, and what its backward pass needs (None unless `save`). `weights` holds
    w_ih, w_hh, b_ih, b_hh of every direction."""
    T, B, I = x.shape
    nd, H3, H = len(weights) // 4, weights[1].shape[0], weights[1].shape[1]
    w_ih = torch.cat(weights[0::4]) if nd > 1 else weights[0]
    b_ih = torch.cat(weights[2::4]) if nd > 1 else weights[2]
    w_hh = [_aligned(w) for w in weights[1::4]]
    b_hh = [b.contiguous() for b in weights[3::4]]
    # input projections of both directions in one GEMM: [T*B, nd*3H]
    gx = torch.addmm(b_ih, x.reshape(T * B, I), w_ih.t())
    y = torch.empty(T, B, nd * H, dtype=torch.float32, device=x.device)
    rsv = torch.empty(nd, T, B, H, 4, dtype=torch.float32, device=x.device) if save else None
    stream = torch.cuda.current_stream(x.device).cuda_stream
    rc = _lib.lib().bc_gru_forward(T, B, H, nd, _ptr(w_hh[0]), _ptr(w_hh[-1]), _ptr(b_hh[0]), _ptr(b_hh[-1]), _ptr(gx), _ptr(y), _ptr(rsv),
                                   _ptr(_scratch(x.device, stream, T, B, H, nd)), _ptr(_status_word(x.device)), _TIMEOUT_S, C.c_void_p(stream))
    _lib.check(rc, "bc_gru_forward")
    global launch_count
    launch_count += 1
    return y, ((x, w_ih, y, rsv, *w_hh) if save else None)


class _GRULayer(torch.autograd.Function):
    """One (bi)directional GRU layer: `apply(x, w_ih, w_hh, b_ih, b_hh[, the same of direction 1])`."""

    @staticmethod
    def forward(ctx, x, *weights):
        y, saved = _forward(x, list(weights), True)
        ctx.save_for_backward(*saved)
        return y

    @staticmethod
    def backward(ctx, dy):
        x, w_ih, y, rsv, *w_hh = ctx.saved_tensors
        T, B, I = x.shape
        nd, H = len(w_hh), w_hh[0].shape[1]
        H3 = 3 * H
        dy = dy.contiguous()
        # gradients of the pre-activations: (dr, dz, dn) of every direction, then dn * r of every direction
        dg = torch.empty(T, B, nd * 4 * H, dtype=torch.float32, device=x.device)
        db = torch.empty(nd, 2, H3, dtype=torch.float32, device=x.device)
        stream = torch.cuda.current_stream(x.device).cuda_stream
        rc = _lib.lib().bc_gru_backward(T, B, H, nd, _ptr(w_hh[0]), _ptr(w_hh[-1]), _ptr(y), _ptr(rsv), _ptr(dy), _ptr(dg), _ptr(db),
                                        _ptr(_scratch(x.device, stream, T, B, H, nd)), _ptr(_status_word(x.device)), _TIMEOUT_S,
                                        C.c_void_p(stream))
        _lib.check(rc, "bc_gru_backward")
        global launch_count
        launch_count += 1
        need = ctx.needs_input_grad
        dgx = dg.view(T * B, nd * 4 * H)[:, :nd * H3]
        dx = (dgx @ w_ih).view(T, B, I) if need[0] else None
        dw_ih = (dgx.t() @ x.reshape(T * B, I)).view(nd, H3, I) if any(need[1::4]) else None
        grads = [dx]
        for d in range(nd):
            dw_hh = None
            if need[2 + 4 * d]:
                dw_hh = torch.empty(H3, H, dtype=torch.float32, device=x.device)
                if T > 1:
                    # direction 0: h_{t-1} = y[t-1]; direction 1 runs backwards in time: h_prev = y[t+1]
                    g = (dg[1:] if d == 0 else dg[:-1]).view(-1, nd * 4 * H)
                    h = (y[:-1] if d == 0 else y[1:])[:, :, d * H:(d + 1) * H].reshape(-1, H)
                    torch.mm(g[:, d * H3:d * H3 + 2 * H].t(), h, out=dw_hh[:2 * H])
                    torch.mm(g[:, nd * H3 + d * H:nd * H3 + (d + 1) * H].t(), h, out=dw_hh[2 * H:])
                else:
                    dw_hh.zero_()
            grads += [dw_ih[d] if need[1 + 4 * d] else None, dw_hh, db[d, 0] if need[3 + 4 * d] else None, db[d, 1] if need[4 + 4 * d] else None]
        return tuple(grads)


def _layer(x: torch.Tensor, weights: List[torch.Tensor]) -> torch.Tensor:
    if torch.is_grad_enabled() and (x.requires_grad or any(w.requires_grad for w in weights)):
        return _GRULayer.apply(x, *weights)
    return _forward(x, weights, False)[0]


def gru_layer(x: torch.Tensor, w_ih: torch.Tensor, w_hh: torch.Tensor, b_ih: torch.Tensor, b_hh: torch.Tensor) -> torch.Tensor:
    """One GRU layer over a time-major fp32 sequence x [T, B, I] with zero initial state.
    Parameters are stacked over the directions (1 or 2). Returns [T, B, ndir * H]."""
    return _layer(x.contiguous(), [t[d] for d in range(w_hh.shape[0]) for t in (w_ih, w_hh, b_ih, b_hh)])


def gru_forward(rnn: torch.nn.GRU, x: torch.Tensor) -> torch.Tensor:
    """`rnn(x)[0]` for a time-major `torch.nn.GRU` with biases and zero initial state, computed by
    the persistent kernels. Raises if the module or the shapes are not supported (use `supported`)."""
    if rnn.batch_first or not rnn.bias or rnn.dropout != 0.0 or getattr(rnn, "proj_size", 0):
        raise ValueError("gru_forward needs a time-major nn.GRU with biases, no dropout and no projection")
    nd = 2 if rnn.bidirectional else 1
    out = x.contiguous()
    for layer in range(rnn.num_layers):
        sfx = (f"_l{layer}", f"_l{layer}_reverse")[:nd]
        out = _layer(out, [getattr(rnn, n + s) for s in sfx for n in ("weight_ih", "weight_hh", "bias_ih", "bias_hh")])
    return out

"""Batch normalisation fused with the clipped ReLU behind it, for training on CUDA.

`BatchNormClip2d` is a `torch.nn.BatchNorm2d` (same parameters, buffers and `state_dict` keys)
whose output is `clamp(bn(x), 0, clip)`. In training mode on contiguous fp32 CUDA activations it
runs the library's two-pass kernels (`csrc/cuda/bn_clip.cu`; the call path is native, `csrc/torch/bindings.cc`): each pass reads its inputs once, so
forward moves 3 and backward 5 tensor sizes through HBM, and the clip mask of the backward pass is
recomputed from the input instead of being stored. Everywhere else (evaluation, CPU, other
dtypes or layouts) it is `F.batch_norm` followed by `F.hardtanh`.

The reference's pieces are FusedBatchNorm on cuDNN and a separate clipping kernel
(tensorflow/core/kernels/fused_batch_norm_op.cu.cc, relu_op_gpu.cu.cc).
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

from .. import _lib


def __getattr__(name):
    if name == "launch_count":   # fused forward and backward calls made by this process
        return int(_lib.ext().bn_launches())
    raise AttributeError(name)


def bn_clip(x, weight, bias, running_mean, running_var, eps: float, momentum: float, clip: float) -> torch.Tensor:
    """Training-mode `clamp(batch_norm(x), 0, clip)` on the fused kernels; `running_mean` /
    `running_var` (or None) are updated in place with weight `momentum` for the new value."""
    return _lib.ext().bn_clip(x, weight, bias, running_mean, running_var, None, eps, momentum, clip)


class BatchNormClip2d(torch.nn.BatchNorm2d):
    """`BatchNorm2d` followed by `Hardtanh(0, clip)` in one module (and, in training on CUDA, in
    two kernels per pass)."""

    def __init__(self, num_features: int, clip: float = 20.0, **kw):
        super().__init__(num_features, **kw)
        self.clip = float(clip)

    def _fused_ok(self, x: torch.Tensor) -> bool:
        return (self.training and x.is_cuda and x.dtype == torch.float32 and x.dim() == 4 and x.is_contiguous() and self.affine
                and self.momentum is not None and (not self.track_running_stats or self._buffers.get("running_mean") is not None)
                and x.numel() > 0 and x.shape[2] * x.shape[3] < 2 ** 31)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        # Parameters and buffers are taken from the module's dictionaries where they are there: an attribute of a module
        # costs most of a microsecond, and a small batch is bound by the host. (A parametrised weight is not there.)
        weight = self._parameters.get("weight")
        if weight is None and self.affine:
            weight = self.weight
        if not self._fused_ok(x) or weight.dtype != torch.float32:
            return F.hardtanh(super().forward(x), 0.0, self.clip)
        bias = self._parameters.get("bias")
        if bias is None:
            bias = self.bias
        # The kernels update the running statistics and the counter of batches.
        b = self._buffers
        rm, rv, count = (b["running_mean"], b["running_var"], b["num_batches_tracked"]) if self.track_running_stats else (None, None, None)
        return _lib.ext().bn_clip(x, weight, bias, rm, rv, count, self.eps, self.momentum, self.clip)

    def extra_repr(self) -> str:
        return super().extra_repr() + f", clip={self.clip}"

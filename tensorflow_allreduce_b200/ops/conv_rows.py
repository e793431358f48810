"""Convolutions of the speech model's front end on the library's tcgen05 kernels.

`RowConv2d` is a `torch.nn.Conv2d` (same parameters and `state_dict` keys). With 32 output channels, vertical stride 2 and
either 32 input channels at horizontal stride 1 or one input channel at horizontal stride 2, fp32 NCHW CUDA tensors and
TF32 convolutions allowed (`torch.backends.cudnn.allow_tf32` or `.conv.fp32_precision`), it runs
`csrc/cuda/conv_rows.cu` forward and backward: the tensors stay
NCHW, TF32 operands are rounded to nearest and sums are fp32. Everything else, other numbers of channels among it, is `F.conv2d`, on the speech model's shapes two to twenty times slower.

The reference's pieces are Conv2D and its gradients on cuDNN (tensorflow/core/kernels/conv_ops.cc, conv_grad_filter_ops.cc,
conv_grad_input_ops.cc).
"""
from __future__ import annotations

import torch

from .. import _lib


def __getattr__(name):
    if name == "launch_count":   # passes (forward, input gradient, weight gradient) run by this process
        return int(_lib.ext().conv_launches())
    raise AttributeError(name)


class RowConv2d(torch.nn.Conv2d):
    """`Conv2d` whose covered forms (see the module's docstring) run on the row convolution kernels."""

    def _covered(self, x: torch.Tensor) -> bool:
        if not (x.is_cuda and x.dim() == 4 and x.numel() > 0) or torch.is_autocast_enabled("cuda"):
            return False
        sw = {32: 1, 1: 2}.get(self.in_channels)
        return (self.out_channels == 32 and sw is not None and self.stride == (2, sw) and self.dilation == (1, 1) and self.groups == 1
                and self.bias is None and self.padding_mode == "zeros" and not isinstance(self.padding, str)
                and _lib.ext().conv_supported(x, self.weight, *self.padding))

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        if not self._covered(x):
            return super().forward(x)
        from .persistent_gru import _ext

        return _ext().conv_rows(x, self.weight, *self.padding)

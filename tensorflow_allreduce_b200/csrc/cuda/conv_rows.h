// 2-D convolutions of the speech model's front end (32 output channels, vertical stride 2) on the 5th-generation tensor
// cores: forward, gradient of the input, gradient of the weight. NCHW fp32 tensors, TF32 operands rounded to nearest, fp32
// accumulation. See conv_rows.cu.
//
// Two forms are covered:
//   32 -> 32 channels, stride (2, 1)     (forward, both gradients)
//   1 -> 32 channels, stride (2, 2)      (forward, gradient of the weight)
//
// The reference's counterparts are Conv2D on cuDNN and its gradients (tensorflow/core/kernels/conv_ops.cc,
// conv_grad_filter_ops.cc, conv_grad_input_ops.cc).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace bc {
namespace gpu {

struct ConvDims {
  int N, Cin, H, W;     // input
  int KH, KW, ph, pw;   // kernel and zero padding; 32 output channels
  int stride_w;         // 1 (Cin 32) or 2 (Cin 1); the vertical stride is 2
  int Ho() const { return (H + 2 * ph - KH) / 2 + 1; }
  int Wo() const { return (W + 2 * pw - KW) / stride_w + 1; }
};

bool conv_rows_supported(const ConvDims& d, int device);
// Bytes of scratch that any of the three passes needs: packed weights, or partial sums of the weight gradient.
size_t conv_rows_scratch_bytes(const ConvDims& d);

// x [N, Cin, H, W], w [32, Cin, KH, KW], y [N, 32, Ho, Wo]; scratch 128-byte aligned. `status`: a word that is ORed with a
// code if a bounded wait inside the kernel ran out (`timeout_s`).
cudaError_t conv_rows_forward(const ConvDims& d, const float* x, const float* w, float* y, void* scratch, uint32_t* status, double timeout_s,
                              cudaStream_t stream);
// Cin = 32 only.
cudaError_t conv_rows_backward_input(const ConvDims& d, const float* dy, const float* w, float* dx, void* scratch, uint32_t* status,
                                     double timeout_s, cudaStream_t stream);
cudaError_t conv_rows_backward_weight(const ConvDims& d, const float* x, const float* dy, float* dw, void* scratch, uint32_t* status,
                                      double timeout_s, cudaStream_t stream);

}  // namespace gpu
}  // namespace bc

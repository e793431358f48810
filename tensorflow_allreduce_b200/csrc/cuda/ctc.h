// CTC loss of a batch whose utterances all have T frames, mean over the batch, and its gradient. The reference computes it on
// the CPU (tensorflow/core/kernels/ctc_loss_op.cc:167, core/util/ctc/ctc_loss_calculator.h).
#pragma once

#include <cuda_runtime.h>

namespace bc {
namespace gpu {

constexpr int kCtcMaxLabels = 511;   // 2 L + 1 states, one thread each

// logp: [T, B, C] log-probabilities; labels: [B, Lmax], rows `stride` apart; lens: [B]; class 0 is the blank.
// chains: [2, B, T, 2 Lmax + 1], log-probabilities of the prefixes (0) and the suffixes (1) up to every state; nll: [B]; loss: [1],
// the mean of nll / max(length, 1), where an utterance without a valid path counts as zero.
cudaError_t ctc_forward(const float* logp, const long long* labels, long long stride, const long long* lens, float* chains, float* nll,
                        float* loss, int T, int B, int C, int Lmax, cudaStream_t stream);

// dlogp: [T, B, C], for a gradient *dloss of the loss.
cudaError_t ctc_backward(const float* logp, const long long* labels, long long stride, const long long* lens, const float* chains,
                         const float* nll, const float* dloss, float* dlogp, int T, int B, int C, int Lmax, cudaStream_t stream);

}  // namespace gpu
}  // namespace bc

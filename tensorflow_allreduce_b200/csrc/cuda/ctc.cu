// CTC loss: the chains of prefixes and suffixes of every utterance, then the gradient (ctc.h).
//
// What bounds it: T dependent steps over 2 L + 1 states that fit into one block. So the prefix and the suffix chain of an utterance
// run beside each other as two blocks of ONE kernel (the suffix chain is the prefix chain of the reversed utterance), a state
// stays in its thread, the neighbours pass through shared memory with one barrier per step, and the log-probabilities of the next
// kAhead steps are on their way while these are added up. The gradient has no chain: a warp per frame, in fixed order (the
// same result in every run). The training step of the speech model (350 frames, 32 utterances of 100 labels) went from 23.8 to
// 22.7 ms with it: torch's kernels were 0.52 ms, one chain after the other, between waits for the device.
#include "ctc.h"

#include <cmath>

namespace bc {
namespace gpu {
namespace {

constexpr int kAhead = 8;          // steps of log-probabilities in flight: a step is about a quarter of a trip to L2
constexpr int kGradWarps = 8;
constexpr int kBlank = 0;

__device__ __forceinline__ int length_of(const long long* lens, int b, int Lmax) {
  return (int)min(max(lens[b], 0ll), (long long)Lmax);
}

__device__ __forceinline__ int class_of(const long long* labels, int l, int C) {
  return (int)min(max(labels[l], 0ll), (long long)(C - 1));
}

__device__ __forceinline__ float log_add(float a, float b, float c) {
  const float m = fmaxf(fmaxf(a, b), c);
  if (m == -INFINITY) return m;
  return m + logf(expf(a - m) + expf(b - m) + expf(c - m));
}

__global__ void __launch_bounds__(1024) ctc_chain_kernel(const float* __restrict__ logp, const long long* __restrict__ labels, long long stride,
                                                         const long long* __restrict__ lens, float* __restrict__ chains,
                                                         float* __restrict__ nll, int T, int B, int C, int Lmax) {
  extern __shared__ float rows[];                          // two rows of states behind two that are never reached
  const int b = blockIdx.x, s = threadIdx.x, width = blockDim.x + 2;
  const bool reversed = blockIdx.y == 1;
  const int L = length_of(lens, b, Lmax), S = 2 * L + 1;
  const bool active = s < S;
  const int state = reversed ? S - 1 - s : s;
  int cls = kBlank;
  bool skip = false;                                       // from the label before, past the blank between them
  labels += b * stride;
  if (active && (s & 1)) {
    const int l = state >> 1;
    cls = class_of(labels, l, C);
    if (s >= 3) skip = labels[l] != labels[reversed ? l + 1 : l - 1];
  }
  if (s < 2) rows[s] = rows[width + s] = -INFINITY;
  const long long step = (long long)(reversed ? -B : B) * C, out_step = reversed ? -(2 * Lmax + 1) : 2 * Lmax + 1;
  const long long first = reversed ? T - 1 : 0;
  const float* lp = logp + (first * B + b) * C + cls;
  float* out = chains + (((long long)blockIdx.y * B + b) * T + first) * (2 * Lmax + 1) + state;

  float now[kAhead], next[kAhead];
#pragma unroll
  for (int j = 0; j < kAhead; j++) next[j] = active && j < T ? lp[j * step] : 0.f;
  float v = -INFINITY;
  for (int i0 = 0; i0 < T; i0 += kAhead) {
#pragma unroll
    for (int j = 0; j < kAhead; j++) {
      now[j] = next[j];
      const int i = i0 + kAhead + j;
      next[j] = active && i < T ? lp[i * step] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < kAhead; j++) {
      const int i = i0 + j;
      if (i >= T) break;
      if (active) {
        if (i == 0) {
          v = s < 2 ? now[j] : -INFINITY;
        } else {
          const float* r = rows + (j & 1 ? 0 : width) + s;   // kAhead is even: the row of step i - 1
          v = log_add(v, r[1], skip ? r[0] : -INFINITY) + now[j];
        }
        out[i * out_step] = v;
      }
      rows[(j & 1 ? width : 0) + 2 + s] = v;
      __syncthreads();
    }
  }
  if (!reversed && s == 0) {
    const float* r = rows + (T & 1 ? 0 : width) + 2;
    nll[b] = -log_add(r[S - 1], S > 1 ? r[S - 2] : -INFINITY, -INFINITY);
  }
}

__global__ void __launch_bounds__(32) ctc_mean_kernel(const float* __restrict__ nll, const long long* __restrict__ lens, float* __restrict__ loss,
                                                      int B, int Lmax) {
  float sum = 0.f;
  for (int b = threadIdx.x; b < B; b += 32) {
    const float v = nll[b];
    sum += v == INFINITY ? 0.f : v / (float)max(length_of(lens, b, Lmax), 1);
  }
#pragma unroll
  for (int d = 16; d > 0; d /= 2) sum += __shfl_xor_sync(~0u, sum, d);
  if (threadIdx.x == 0) *loss = sum / (float)B;
}

// Gradient of -log p with respect to a log-probability, for log-probabilities that come out of a softmax: what the class
// weighs in the frame less what the paths through it weigh.
__global__ void __launch_bounds__(32 * kGradWarps) ctc_grad_kernel(const float* __restrict__ logp, const long long* __restrict__ labels,
                                                                   long long stride, const long long* __restrict__ lens,
                                                                   const float* __restrict__ chains, const float* __restrict__ nll,
                                                                   const float* __restrict__ dloss, float* __restrict__ dlogp, int T, int B, int C,
                                                                   int Lmax) {
  extern __shared__ int shared[];
  const int b = blockIdx.y, warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int L = length_of(lens, b, Lmax), S = 2 * L + 1, width = 2 * Lmax + 1;
  int* lab = shared;
  float* weight = reinterpret_cast<float*>(shared) + (1 + warp) * Lmax;
  for (int l = threadIdx.x; l < L; l += blockDim.x) lab[l] = class_of(labels + b * stride, l, C);
  __syncthreads();
  const int t = blockIdx.x * kGradWarps + warp;
  if (t >= T) return;
  const float* lp = logp + ((long long)t * B + b) * C;
  float* out = dlogp + ((long long)t * B + b) * C;
  const float n = nll[b];
  if (n == INFINITY) {                                     // no path: no gradient
    for (int k = lane; k < C; k += 32) out[k] = 0.f;
    return;
  }
  const float scale = *dloss / (float)B / (float)max(L, 1);
  const float* alpha = chains + ((long long)b * T + t) * width;
  const float* beta = alpha + (long long)B * T * width;
  float blank = 0.f, all = 0.f;
  for (int s = lane; s < S; s += 32) {                     // a lane's states are all blanks or all labels
    const float both = alpha[s] + beta[s];
    const float w = both == -INFINITY ? 0.f : expf(both + n - lp[s & 1 ? lab[s >> 1] : kBlank]);
    if (s & 1) weight[s >> 1] = w;
    else blank += w;
    all += w;
  }
#pragma unroll
  for (int d = 16; d > 0; d /= 2) {
    blank += __shfl_xor_sync(~0u, blank, d);
    all += __shfl_xor_sync(~0u, all, d);
  }
  __syncwarp();
  // The weights of a frame add up to one but for the rounding of its sums of logarithms, which all of them share.
  const float norm = all > 0.f ? 1.f / all : 1.f;
  for (int k = lane; k < C; k += 32) {
    float sum = k == kBlank ? blank : 0.f;
    for (int l = 0; l < L; l++) sum += lab[l] == k ? weight[l] : 0.f;
    out[k] = (expf(lp[k]) - sum * norm) * scale;
  }
}

bool valid(int T, int B, int C, int Lmax) { return T > 0 && B > 0 && B <= 65535 && C > 0 && Lmax >= 0 && Lmax <= kCtcMaxLabels; }

}  // namespace

cudaError_t ctc_forward(const float* logp, const long long* labels, long long stride, const long long* lens, float* chains, float* nll,
                        float* loss, int T, int B, int C, int Lmax, cudaStream_t stream) {
  if (!valid(T, B, C, Lmax)) return cudaErrorInvalidValue;
  const int threads = (2 * Lmax + 1 + 31) / 32 * 32;
  ctc_chain_kernel<<<dim3(B, 2), threads, 2 * (threads + 2) * sizeof(float), stream>>>(logp, labels, stride, lens, chains, nll, T, B, C, Lmax);
  ctc_mean_kernel<<<1, 32, 0, stream>>>(nll, lens, loss, B, Lmax);
  return cudaGetLastError();
}

cudaError_t ctc_backward(const float* logp, const long long* labels, long long stride, const long long* lens, const float* chains,
                         const float* nll, const float* dloss, float* dlogp, int T, int B, int C, int Lmax, cudaStream_t stream) {
  if (!valid(T, B, C, Lmax)) return cudaErrorInvalidValue;
  ctc_grad_kernel<<<dim3((T + kGradWarps - 1) / kGradWarps, B), 32 * kGradWarps, (1 + kGradWarps) * Lmax * sizeof(float), stream>>>(
      logp, labels, stride, lens, chains, nll, dloss, dlogp, T, B, C, Lmax);
  return cudaGetLastError();
}

}  // namespace gpu
}  // namespace bc

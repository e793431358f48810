// Training-mode batch normalisation over NCHW fp32 activations fused with the clipped ReLU that
// follows it in the DeepSpeech2-style model: y = clamp(gamma * (x - mean) / sqrt(var + eps) + beta, 0, hi).
//
// The reference's counterpart is FusedBatchNorm (cuDNN's batch normalisation plus two helper
// kernels, tensorflow/core/kernels/fused_batch_norm_op.cu.cc:26-60) followed by a separate
// Relu6-style clipping kernel (core/kernels/relu_op_gpu.cu.cc). On B200 cuDNN's backward kernel
// for these shapes (32 channels, 0.9 M elements per channel) runs at a twentieth of the memory
// roofline; the two passes here read each tensor twice and write it once, nothing more:
//   forward : pass 1 per-channel sum and sum of squares,
//             pass 2 normalise + scale + shift + clip, save mean / rstd, update the running statistics
//   backward: pass 1 per-channel sums of dz and dz * xhat, where dz = dy inside the clip range
//             (recomputed from x, so the forward output is not needed), pass 2
//             dx = gamma * rstd * (dz - mean(dz) - xhat * mean(dz * xhat)); dgamma, dbeta.
//
// Both passes are bound by memory. What the kernels do about it:
//   * One wave of equal blocks: a channel's N x HW elements are cut into as many contiguous ranges as fill
//     the GPU once (a block per plane left the second of two waves nearly empty).
//   * 16-byte accesses whatever the plane size: a range is peeled to the next 16-byte boundary.
//   * Pass 2 walks every range backwards, so that it starts with what pass 1 read last and L2 still holds: of [32, 32, 81, 350]
//     (116 MB) it reads 51 of 116 MB from memory forward and 150 of 232 backward; walking forwards 63.8 / 105.5 us instead of
//     61.6 / 101.4.
//   * The sums of a block are stored, not added up atomically: no memory to clear beforehand, and results that are
//     the same in every run. Every block of pass 2 adds up its channel's few.
//   * Pass 2 is launched early (programmatic dependent launch) and waits on the device for the end of pass 1.
// [32, 32, 81, 350], forward 3, backward 5 passes over it: 61.6 / 101.4 us for the two kernels each, 5.7 TB/s of what passes.
#include "bn_clip.h"

#include <stdint.h>

#include <algorithm>
#include <initializer_list>

namespace bc {
namespace gpu {

namespace {

constexpr int kThreads = 256;
// [32, 32, 81, 350], forward / backward us: 2 blocks 65.4 / 101.3, 4 blocks 61.4 / 101.4, 6 blocks 73.3 / 113.7, 8 blocks 84.3 / 130.1 (too few
// registers for the loads in flight); [32, 32, 41, 175]: 27.4 / 33.8, 24.5 / 29.7, 28.8 / 37.9, 33.4 / 42.0.
constexpr int kBlocksPerSm = 4;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum of two per-thread values over the block, stored by thread 0.
__device__ __forceinline__ void block_sum2(float a, float b, double2* out) {
  __shared__ float sa[kThreads / 32], sb[kThreads / 32];
  a = warp_sum(a);
  b = warp_sum(b);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { sa[w] = a; sb[w] = b; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double x = 0.0, y = 0.0;
#pragma unroll
    for (int i = 0; i < kThreads / 32; i++) { x += sa[i]; y += sb[i]; }
    *out = make_double2(x, y);
  }
}

// Sum of a channel's n partial sums, the same in every thread of the block.
__device__ __forceinline__ double2 channel_sum(const double2* part, int n) {
  __shared__ double2 total;
  if (threadIdx.x < 32) {
    double x = 0.0, y = 0.0;
    for (int i = threadIdx.x; i < n; i += 32) {
      const double2 v = __ldcg(part + i);
      x += v.x;
      y += v.y;
    }
    x = warp_sum(x);
    y = warp_sum(y);
    if (threadIdx.x == 0) total = make_double2(x, y);
  }
  __syncthreads();
  return total;
}

// The elements of channel blockIdx.y that block blockIdx.x works on: [lo, hi) of the N x HW elements of the channel counted
// image by image. They lie in one piece per image. `piece(first, len)` is called for each: in order, or backwards
// (REVERSE), by the whole block, or (WARPS) by one warp each where an image's plane is short.
template <bool WARPS, bool REVERSE, typename F>
__device__ __forceinline__ void for_pieces(int N, int C, int HW, F piece) {
  const size_t m = (size_t)N * HW;
  size_t share = (m + gridDim.x - 1) / gridDim.x;
  share = (share + 3) & ~(size_t)3;
  const size_t lo = blockIdx.x * share;
  if (lo >= m) return;
  const size_t hi = lo + share < m ? lo + share : m;
  const int n0 = (int)(lo / HW), n1 = (int)((hi - 1) / HW), c = blockIdx.y;
  for (int k = WARPS ? threadIdx.x >> 5 : 0; k <= n1 - n0; k += WARPS ? kThreads / 32 : 1) {
    const int n = REVERSE ? n1 - k : n0 + k;
    const int from = n == n0 ? (int)(lo - (size_t)n0 * HW) : 0, to = n == n1 ? (int)(hi - (size_t)n1 * HW) : HW;
    piece(((size_t)n * C + c) * HW + from, to - from);
  }
}

// One piece, elements [first, first + len) of the tensor: `vec(i)` for U 16-byte vectors at element i, i + stride, ... at a
// time (`n` of them exist), `one(i)` for the elements before the first and behind the last 16-byte boundary (VEC: the
// tensors start on such boundaries; otherwise for all).
template <bool WARPS, bool REVERSE, bool VEC, int U, typename FV, typename F1>
__device__ __forceinline__ void for_vectors(size_t first, int len, FV vec, F1 one) {
  constexpr int S = WARPS ? 32 : kThreads;
  const int t = WARPS ? threadIdx.x & 31 : threadIdx.x;
  const int head = VEC ? min(len, (int)((4 - (first & 3)) & 3)) : len;
  const int nvec = (len - head) >> 2;
  const size_t v0 = first + head;
  const int chunks = (nvec + S * U - 1) / (S * U);
  for (int k = 0; k < chunks; k++) {
    const int at = (REVERSE ? chunks - 1 - k : k) * (S * U) + t;
    vec(v0 + (size_t)at * 4, S * 4, nvec - at <= 0 ? 0 : (nvec - at + S - 1) / S);
  }
  for (int i = t; i < head; i += S) one(first + i);
  for (int i = nvec * 4 + t; i < len - head; i += S) one(v0 + i);
}

// Forward pass 1: part[channel][block] = sum x, sum x^2 over the block's range.
template <bool WARPS, bool VEC>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm) bn_stats_kernel(const float* __restrict__ x, double2* __restrict__ part, int N, int C, int HW) {
  cudaTriggerProgrammaticLaunchCompletion();
  constexpr int U = 8;
  float s[4] = {}, q[4] = {};
  for_pieces<WARPS, false>(N, C, HW, [&](size_t first, int len) {
    for_vectors<WARPS, false, VEC, U>(
        first, len,
        [&](size_t i, int stride, int n) {
          float4 a[U];
#pragma unroll
          for (int u = 0; u < U; u++) a[u] = u < n ? *reinterpret_cast<const float4*>(x + i + u * stride) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int u = 0; u < U; u++) {
            s[0] += a[u].x; q[0] = fmaf(a[u].x, a[u].x, q[0]);
            s[1] += a[u].y; q[1] = fmaf(a[u].y, a[u].y, q[1]);
            s[2] += a[u].z; q[2] = fmaf(a[u].z, a[u].z, q[2]);
            s[3] += a[u].w; q[3] = fmaf(a[u].w, a[u].w, q[3]);
          }
        },
        [&](size_t i) { s[0] += x[i]; q[0] = fmaf(x[i], x[i], q[0]); });
  });
  block_sum2((s[0] + s[1]) + (s[2] + s[3]), (q[0] + q[1]) + (q[2] + q[3]), part + (size_t)blockIdx.y * gridDim.x + blockIdx.x);
}

// Forward pass 2. The first block of every channel also publishes the batch statistics and
// folds them into the running ones.
template <bool WARPS, bool VEC>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm) bn_apply_kernel(const float* __restrict__ x, float* __restrict__ y, const double2* __restrict__ part,
                                                                         const float* __restrict__ gamma, const float* __restrict__ beta,
                                                                         float* __restrict__ save_mean, float* __restrict__ save_rstd,
                                                                         float* running_mean, float* running_var, long long* batches, int N, int C, int HW, float eps,
                                                                         float momentum, float clip_hi) {
  cudaGridDependencySynchronize();
  const int c = blockIdx.y;
  const double2 acc = channel_sum(part + (size_t)c * gridDim.x, gridDim.x);
  const double m = (double)N * HW;
  const double mean_d = acc.x / m;
  double var_d = acc.y / m - mean_d * mean_d;
  if (var_d < 0.0) var_d = 0.0;
  const float mean = (float)mean_d;
  const float rstd = rsqrtf((float)var_d + eps);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    save_mean[c] = mean;
    save_rstd[c] = rstd;
    if (batches && c == 0) *batches += 1;
    if (running_mean) {
      const float unbiased = (float)(var_d * (m / (m > 1.0 ? m - 1.0 : 1.0)));
      running_mean[c] = (1.f - momentum) * running_mean[c] + momentum * mean;
      running_var[c] = (1.f - momentum) * running_var[c] + momentum * unbiased;
    }
  }
  const float scale = gamma[c] * rstd;
  const float shift = beta[c] - mean * scale;
  auto f = [&](float v) { return fminf(fmaxf(fmaf(v, scale, shift), 0.f), clip_hi); };
  constexpr int U = 8;
  for_pieces<WARPS, true>(N, C, HW, [&](size_t first, int len) {
    for_vectors<WARPS, true, VEC, U>(
        first, len,
        [&](size_t i, int stride, int n) {
          float4 a[U];
#pragma unroll
          for (int u = 0; u < U; u++)
            if (u < n) a[u] = __ldcs(reinterpret_cast<const float4*>(x + i + u * stride));
#pragma unroll
          for (int u = 0; u < U; u++)
            if (u < n) __stcs(reinterpret_cast<float4*>(y + i + u * stride), make_float4(f(a[u].x), f(a[u].y), f(a[u].z), f(a[u].w)));
        },
        [&](size_t i) { y[i] = f(x[i]); });
  });
}

// dz of one element: dy where the pre-clip value lies strictly inside (0, hi), else 0 (the
// gradient rule of a hard clamp).
__device__ __forceinline__ float masked(float dy, float z, float clip_hi) { return (z > 0.f && z < clip_hi) ? dy : 0.f; }

// Backward pass 1: part[channel][block] = sum dz, sum dz * xhat.
template <bool WARPS, bool VEC>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm) bn_bwd_reduce_kernel(const float* __restrict__ x, const float* __restrict__ dy,
                                                                              const float* __restrict__ gamma, const float* __restrict__ beta,
                                                                              const float* __restrict__ save_mean, const float* __restrict__ save_rstd,
                                                                              double2* __restrict__ part, int N, int C, int HW, float clip_hi) {
  cudaTriggerProgrammaticLaunchCompletion();
  const int c = blockIdx.y;
  const float mean = save_mean[c], rstd = save_rstd[c], g = gamma[c], b = beta[c];
  constexpr int U = 4;
  float s1[4] = {}, s2[4] = {};
  auto f = [&](float xv, float dv, int e) {
    const float h = (xv - mean) * rstd;
    const float z = masked(dv, fmaf(h, g, b), clip_hi);
    s1[e] += z;
    s2[e] = fmaf(z, h, s2[e]);
  };
  for_pieces<WARPS, false>(N, C, HW, [&](size_t first, int len) {
    for_vectors<WARPS, false, VEC, U>(
        first, len,
        [&](size_t i, int stride, int n) {
          float4 a[U], d[U];
#pragma unroll
          for (int u = 0; u < U; u++) {
            a[u] = u < n ? *reinterpret_cast<const float4*>(x + i + u * stride) : make_float4(0.f, 0.f, 0.f, 0.f);
            d[u] = u < n ? *reinterpret_cast<const float4*>(dy + i + u * stride) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
#pragma unroll
          for (int u = 0; u < U; u++) { f(a[u].x, d[u].x, 0); f(a[u].y, d[u].y, 1); f(a[u].z, d[u].z, 2); f(a[u].w, d[u].w, 3); }
        },
        [&](size_t i) { f(x[i], dy[i], 0); });
  });
  block_sum2((s1[0] + s1[1]) + (s1[2] + s1[3]), (s2[0] + s2[1]) + (s2[2] + s2[3]), part + (size_t)c * gridDim.x + blockIdx.x);
}

// Backward pass 2.
template <bool WARPS, bool VEC>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm) bn_bwd_apply_kernel(const float* __restrict__ x, const float* __restrict__ dy, float* __restrict__ dx,
                                                                             const float* __restrict__ gamma, const float* __restrict__ beta,
                                                                             const float* __restrict__ save_mean, const float* __restrict__ save_rstd,
                                                                             const double2* __restrict__ part, float* __restrict__ dgamma,
                                                                             float* __restrict__ dbeta, int N, int C, int HW, float clip_hi) {
  const int c = blockIdx.y;
  const float mean = save_mean[c], rstd = save_rstd[c], g = gamma[c], b = beta[c];
  cudaGridDependencySynchronize();
  const double2 acc = channel_sum(part + (size_t)c * gridDim.x, gridDim.x);
  const double m = (double)N * HW;
  const float s1 = (float)(acc.x / m), s2 = (float)(acc.y / m);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    dbeta[c] = (float)acc.x;
    dgamma[c] = (float)acc.y;
  }
  const float k = g * rstd;
  auto f = [&](float xv, float dv) {
    const float h = (xv - mean) * rstd;
    const float z = masked(dv, fmaf(h, g, b), clip_hi);
    return k * (z - s1 - h * s2);
  };
  constexpr int U = 4;
  for_pieces<WARPS, true>(N, C, HW, [&](size_t first, int len) {
    for_vectors<WARPS, true, VEC, U>(
        first, len,
        [&](size_t i, int stride, int n) {
          float4 a[U], d[U];
#pragma unroll
          for (int u = 0; u < U; u++)
            if (u < n) {
              a[u] = __ldcs(reinterpret_cast<const float4*>(x + i + u * stride));
              d[u] = __ldcs(reinterpret_cast<const float4*>(dy + i + u * stride));
            }
#pragma unroll
          for (int u = 0; u < U; u++)
            if (u < n)
              __stcs(reinterpret_cast<float4*>(dx + i + u * stride),
                     make_float4(f(a[u].x, d[u].x), f(a[u].y, d[u].y), f(a[u].z, d[u].z), f(a[u].w, d[u].w)));
        },
        [&](size_t i) { dx[i] = f(x[i], dy[i]); });
  });
}

int sm_count_of_current_device() {
  int dev = 0, n = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

// Blocks per channel: what fills the GPU once, but no block with less than four elements per thread.
int blocks_per_channel(int N, int C, int HW) {
  const long fill = std::min(sm_count_of_current_device(), kBnMaxSms) * kBlocksPerSm / C;
  const long most = (long)(((long long)N * HW + 4 * kThreads - 1) / (4 * kThreads));
  return (int)std::max(1L, std::min(fill, most));
}

bool aligned16(std::initializer_list<const void*> ptrs) {
  for (const void* p : ptrs)
    if (((uintptr_t)p & 15) != 0) return false;
  return true;
}

// Planes of fewer elements than this are given to single warps (a block needs 1024 for one vector per thread). 32 images of 32
// channels, us, warps / blocks: planes of 221 forward 13.5 / 23.8, backward 13.3 / 23.6; 780: 14.2 / 17.3, 15.4 / 17.4; 1681: 16.2 / 19.7,
// 19.5 / 21.5; 2460: 16.9 / 17.6, 21.5 / 19.5; 3280: 18.3 / 18.0, 25.6 / 19.5; 4100: 19.2 / 19.2, 29.7 / 23.3; 5248: 21.3 / 19.4, 33.8 / 23.6.
// The line is that of the forward pass; the backward pass would have it at 2000.
constexpr int kShortPlane = 4096;

template <typename K, typename... A>
cudaError_t launch(bool dependent, K kernel, dim3 grid, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kThreads);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <bool WARPS, bool VEC>
cudaError_t forward(const float* x, float* y, const float* gamma, const float* beta, float* running_mean, float* running_var, long long* batches, float* save_mean,
                    float* save_rstd, double2* part, int N, int C, int HW, float eps, float momentum, float clip_hi, cudaStream_t stream) {
  const dim3 grid(blocks_per_channel(N, C, HW), C);
  cudaError_t e = launch(false, bn_stats_kernel<WARPS, VEC>, grid, stream, x, part, N, C, HW);
  if (e != cudaSuccess) return e;
  return launch(true, bn_apply_kernel<WARPS, VEC>, grid, stream, x, y, (const double2*)part, gamma, beta, save_mean, save_rstd, running_mean,
                running_var, batches, N, C, HW, eps, momentum, clip_hi);
}

template <bool WARPS, bool VEC>
cudaError_t backward(const float* x, const float* dy, const float* gamma, const float* beta, const float* save_mean, const float* save_rstd, float* dx,
                     float* dgamma, float* dbeta, double2* part, int N, int C, int HW, float clip_hi, cudaStream_t stream) {
  const dim3 grid(blocks_per_channel(N, C, HW), C);
  cudaError_t e = launch(false, bn_bwd_reduce_kernel<WARPS, VEC>, grid, stream, x, dy, gamma, beta, save_mean, save_rstd, part, N, C, HW, clip_hi);
  if (e != cudaSuccess) return e;
  return launch(true, bn_bwd_apply_kernel<WARPS, VEC>, grid, stream, x, dy, dx, gamma, beta, save_mean, save_rstd, (const double2*)part, dgamma,
                dbeta, N, C, HW, clip_hi);
}

}  // namespace

cudaError_t bn_clip_forward(const float* x, float* y, const float* gamma, const float* beta, float* running_mean, float* running_var,
                            long long* batches, float* save_mean, float* save_rstd, double* acc, int N, int C, int HW, float eps, float momentum,
                            float clip_hi, cudaStream_t stream) {
  if (N <= 0 || C <= 0 || HW <= 0 || C > 65535) return cudaErrorInvalidValue;
  const bool vec = aligned16({x, y}), warps = HW < kShortPlane;
  auto fn = warps ? (vec ? forward<true, true> : forward<true, false>) : (vec ? forward<false, true> : forward<false, false>);
  return fn(x, y, gamma, beta, running_mean, running_var, batches, save_mean, save_rstd, (double2*)acc, N, C, HW, eps, momentum, clip_hi, stream);
}

cudaError_t bn_clip_backward(const float* x, const float* dy, const float* gamma, const float* beta, const float* save_mean,
                             const float* save_rstd, float* dx, float* dgamma, float* dbeta, double* acc, int N, int C, int HW,
                             float clip_hi, cudaStream_t stream) {
  if (N <= 0 || C <= 0 || HW <= 0 || C > 65535) return cudaErrorInvalidValue;
  const bool vec = aligned16({x, dy, dx}), warps = HW < kShortPlane;
  auto fn = warps ? (vec ? backward<true, true> : backward<true, false>) : (vec ? backward<false, true> : backward<false, false>);
  return fn(x, dy, gamma, beta, save_mean, save_rstd, dx, dgamma, dbeta, (double2*)acc, N, C, HW, clip_hi, stream);
}

}  // namespace gpu
}  // namespace bc

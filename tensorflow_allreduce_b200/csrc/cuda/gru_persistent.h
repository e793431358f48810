// Persistent bidirectional GRU layer for sm_100a: the recurrent weights of a layer stay on chip (tensor
// memory, and shared memory for what does not fit) for all time steps, the per-step recurrent product runs
// on the 5th-generation tensor cores (tcgen05.mma, fp16 pairs forward, TF32 backward, fp32 accumulator), and the
// two directions run side by side in one cooperative launch. gru_forward.cu, gru_backward.cu: the kernels.
//
// The reference's speech-model pieces are GRU cells that launch one GEMM plus elementwise
// kernels per time step (tensorflow/contrib/rnn/kernels/gru_ops.h:69-119, gru_ops_gpu.cu.cc) or
// cuDNN's RNN (contrib/cudnn_rnn/kernels/cudnn_rnn_ops.cc:738-1091); on B200 that is about
// 7000 launches of 9 us per training step of the DeepSpeech2-style benchmark model.
//
// Gate equations (PyTorch / cuDNN form, gate order r, z, n):
//   r = sigmoid(gx_r + W_hr h + b_hr)      z = sigmoid(gx_z + W_hz h + b_hz)
//   n = tanh(gx_n + r * (W_hn h + b_hn))   h' = n + z * (h - n)
// where gx = W_i x + b_i for all time steps is computed beforehand by one large library GEMM.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace bc {
namespace gpu {

struct GruDims {
  int T;        // time steps
  int B;        // batch, 1..32
  int H;        // hidden size per direction: multiple of 128, at most 1024
  int ndir;     // 1 or 2 (direction 1 runs the sequence backwards)
};

// Status bits written to status[0] by a block whose bounded wait ran out (the kernel then
// returns early; outputs are incomplete).
constexpr uint32_t kGruTimeoutGrid = 1u;      // waiting for the other blocks of its direction
constexpr uint32_t kGruTimeoutBlock = 2u;     // waiting for other warps of the block
constexpr uint32_t kGruTimeoutMma = 4u;       // waiting for the tensor core to finish

// Forward. All tensors are fp32, contiguous, on the current device; w_hh, rsv, fac and scratch 16-byte aligned.
//   w_hh[dir] [3H, H]          recurrent weights of each direction
//   b_hh[dir] [3H]
//   gx    [T, B, ndir, 3H]     input projections including b_ih
//   y     [T, B, ndir*H]       output
// For the backward pass, one of these or none:
//   rsv   [ndir, T, B, H, 4]   r, z, n and (W_hn h + b_hn) of every step
//   fac   [ndir, T, B, 5, H]   what dh is multiplied with to give dr, dz, dn r, dn and its share in the step before
//   scratch                    gru_persistent_scratch_bytes(d) bytes, zeroed once when they are allocated and then reused
//                              as they are by later calls, one after the other (concurrent calls need one each)
//   status[1] uint32           ORed with kGruTimeout* on failure
// `timeout_s` bounds every wait inside the kernel. Returns cudaErrorInvalidValue for unsupported
// dimensions and cudaErrorCooperativeLaunchTooLarge if the grid cannot be co-resident.
cudaError_t gru_persistent_forward(const GruDims& d, const float* const* w_hh, const float* const* b_hh, const float* gx, float* y,
                                   float* rsv, float* fac, void* scratch, uint32_t* status, double timeout_s, cudaStream_t stream);

// Backward through time.
//   y, rsv or fac              from the forward pass; `fac` is the faster one (dh travels between the blocks instead of three gradients either way,
//                              but with `rsv` every block of a group forms the factors of its whole range), y is not read beside it
//   dy     [T, B, ndir*H]      gradient of the output
//   dg     [T, B, ndir*4H]     out: gradients of the pre-activations. Columns [0, ndir*3H): those of gx, (dr, dz, dn) of
//                              direction 0, then of direction 1; columns ndir*3H + dir*H: dn * r. The gradient of
//                              (W_h h + b_h) is (dr, dz, dn * r), so the two share their first two parts.
//   db     [ndir, 2, 3H]       out: sums over time and batch of (dr, dz, dn) and of (dr, dz, dn * r): gradients of b_ih and b_hh
// The caller forms dW_ih, dx and dW_hh from dg with library GEMMs.
cudaError_t gru_persistent_backward(const GruDims& d, const float* const* w_hh, const float* y, const float* rsv, const float* fac, const float* dy,
                                    float* dg, float* db, void* scratch, uint32_t* status, double timeout_s, cudaStream_t stream);

// An upper bound of the bytes of partial sums (plain fp32) that one step exchanges, and the bytes of scratch memory that a forward or
// backward call needs for these dimensions.
size_t gru_persistent_workspace_bytes(const GruDims& d);
size_t gru_persistent_scratch_bytes(const GruDims& d);

// Tuning aid: when `stamps` (device memory, 8 x T uint64) is non-null, thread 0 of block (0, 0) of every later
// launch records %globaltimer at fixed points of each step. Forward: [0] step start, [1] accumulator complete, [2] read back, [3] published, [4] outputs stored, [5] paused,
// [6] its words in shared memory. Backward: [0] step start, [4] published, [1] accumulator complete, [2] partial sums sent, [3] received. Null switches it off.
void gru_persistent_set_profile(unsigned long long* stamps);

// True if this device and these dimensions can run the persistent kernels.
bool gru_persistent_supported(const GruDims& d, int device);

}  // namespace gpu
}  // namespace bc

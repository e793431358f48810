// What the forward and the backward kernel of the persistent GRU layer share: parameters, the words that travel between blocks, the start of
// a launch.
#pragma once

#include "gru_persistent.h"

#include "tcgen05_prims.cuh"

namespace bc {
namespace gpu {
namespace gru {

using namespace tc;

constexpr int kUnits = 16;            // hidden units per block
constexpr uint32_t kTmemCols = 512;
constexpr int kMinSmem = 120 * 1024;  // more than half of an SM's shared memory: one block per SM, since a block takes all of tensor memory

struct Params {
  GruDims d;
  const float* w_hh[2];   // [3H, H] of each direction
  const float* b_hh[2];   // forward: [3H] of each direction
  const float* gx;        // forward
  float* y;               // forward: out; backward: in (const)
  float4* rsv;            // forward: out, or null; backward: in, where there are no factors
  float* fac;             // forward: out, or null; backward: in, or null
  const float* dy;        // backward
  float* dg;              // backward: out
  float* db;              // backward: out
  uint32_t* ring;         // what travels between blocks: operand words, behind them the partial sums of the backward pass
  uint32_t* sync;         // per direction: arrivals, generation
  uint32_t* status;
  unsigned long long timeout_ns;
  unsigned long long* prof;   // optional: 8 time stamps per step of block (0, 0), for tuning
};

__device__ __forceinline__ uint32_t clock32() {
  uint32_t c;
  asm volatile("mov.u32 %0, %%clock;" : "=r"(c));
  return c;
}
// 32 bytes per request: a strong load costs L2 the same whatever its width (fresh lines, 32 KB per block and 128 blocks:
// 1406 cycles this way, 1758 with 16-byte loads).
struct Words { uint32_t w[8]; };
// Two neighbouring chunks of a swizzled row: the second one's place differs in bit 4.
__device__ __forceinline__ void st_shared2(uint32_t at, const Words& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v.w[0]), "r"(v.w[1]), "r"(v.w[2]), "r"(v.w[3]) : "memory");
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at ^ 16), "r"(v.w[4]), "r"(v.w[5]), "r"(v.w[6]), "r"(v.w[7]) : "memory");
}
__device__ __forceinline__ void ld_words(const uint32_t* p, Words& v) {
  asm volatile("ld.relaxed.gpu.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]), "=r"(v.w[6]), "=r"(v.w[7]) : "l"(p) : "memory");
}

// mbar_wait() of a whole warp on the chain of a step. All of it is uniform control flow (see the MMA warp), and the clock, which takes long to
// read, is looked at only by a wait that lasts.
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, unsigned long long timeout_ns, const volatile int* abort_flag) {
  uint32_t spins = 0;
  unsigned long long t0 = 0;
  while (!__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) {
    if (((++spins) & 15) == 0) {
      const unsigned long long now = gtimer();
      if (t0 == 0) t0 = now;
      if (__any_sync(0xffffffffu, *abort_flag != 0 || now - t0 > timeout_ns)) return false;
    }
  }
  return true;
}

// The same for lanes that may have given up one by one.
__device__ __forceinline__ bool lane_wait(uint32_t bar, uint32_t parity, unsigned long long timeout_ns, const volatile int* abort_flag) {
  uint32_t spins = 0;
  unsigned long long t0 = 0;
  while (!mbar_try_wait(bar, parity)) {
    if (((++spins) & 15) == 0) {
      const unsigned long long now = gtimer();
      if (t0 == 0) t0 = now;
      if ((abort_flag && *abort_flag) || now - t0 > timeout_ns) return false;
    }
  }
  return true;
}

// What dh is multiplied with to give the gradients of the pre-activations dr, dz, dn r and dn, and dh's share in the step before.
struct Factors { float r, z, nr, n, keep; };
// From r, z, n and hn = W_hn h + b_hn of a step and h of the step before.
__device__ __forceinline__ Factors factors(float4 v, float hp) {
  const float r = v.x, z = v.y, n = v.z, hn = v.w, c = (1.f - z) * (1.f - n * n);
  return {c * hn * r * (1.f - r), (hp - n) * z * (1.f - z), c * r, c, z};
}

// The blocks of a direction meet once, at the start of a launch: thread 0 of each arrives, and leaves when all have.
struct Meeting {
  uint32_t* count;
  volatile uint32_t* generation;
  uint32_t mine;
};
__device__ __forceinline__ Meeting meet_arrive(const Params& p, int dir, uint32_t blocks) {
  Meeting m{p.sync + dir * 32, p.sync + dir * 32 + 16, 0};
  m.mine = *m.generation;               // read before this block's arrival: cannot move on until it has arrived
  __threadfence();
  if (atomicAdd(m.count, 1u) == blocks - 1) {
    *(volatile uint32_t*)m.count = 0;
    __threadfence();
    *m.generation = m.mine + 1;
  }
  return m;
}
__device__ __forceinline__ bool meet_wait(const Params& p, const Meeting& m) {
  const unsigned long long t0 = gtimer();
  uint32_t spins = 0;
  bool ok = true;
  while (*m.generation == m.mine) {
    if (((++spins) & 31) == 0 && gtimer() - t0 > p.timeout_ns) {
      ok = false;
      atomicOr(p.status, kGruTimeoutGrid);
      break;
    }
  }
  __threadfence();
  return ok;
}

cudaError_t launch_forward(const Params& p, cudaStream_t stream);
cudaError_t launch_backward(const Params& p, cudaStream_t stream);

}  // namespace gru
}  // namespace gpu
}  // namespace bc

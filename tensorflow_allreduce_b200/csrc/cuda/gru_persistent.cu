// Host side of the persistent GRU layer: dimensions, exchange memory, launches. The kernels are in gru_forward.cu and gru_backward.cu.
#include "gru_common.cuh"

#include <algorithm>

namespace bc {
namespace gpu {

namespace {

using namespace gru;

unsigned long long* g_prof = nullptr;   // set by gru_persistent_set_profile()

bool dims_ok(const GruDims& d) {
  return d.T >= 1 && d.T < 4096 && d.B >= 1 && d.B <= 32 && d.H >= 128 && d.H <= 1024 && d.H % 128 == 0 && (d.ndir == 1 || d.ndir == 2);
}

bool aligned(const void* p, uintptr_t bytes) { return ((uintptr_t)p & (bytes - 1)) == 0; }

// Bytes of partial sums (fp32, 32 batch rows, a block's own included) of a step with groups of 4 blocks forward and 16 backward, wider
// than any that is launched.
size_t exchange_bytes(const GruDims& d) {
  const size_t blocks = (size_t)d.ndir * (d.H / kUnits);
  const int widest = d.H / kUnits % 16 == 0 ? 16 : 8;
  return blocks * 32 * 4 * std::max(4 * 3 * kUnits, widest * kUnits);
}
constexpr size_t kSyncBytes = 1024;
// Room for both slots of three words per unit and batch entry and a little more; the backward pass, the larger one, uses one word.
size_t ring_bytes(const GruDims& d) { return (size_t)d.ndir * 2 * (3 * d.H + 16 * 16) * 32 * 4; }
// Rows of partial sums that a block has room for: of groups of four blocks, or of eight where the pass needs them.
int exchange_rows(const GruDims& d) {
  const bool small = d.B <= 16;
  return std::max((d.H <= (small ? 512 : 256) ? 1 : 2) * 3 * kUnits, (d.H <= (small ? 256 : 512) ? 4 : 8) * kUnits);
}

cudaError_t start(Params& p, const GruDims& d, const float* const* w_hh, void* scratch, uint32_t* status, double timeout_s) {
  // factors and words of the ring are read 32 bytes at a time
  if (!dims_ok(d) || !aligned(p.rsv, 16) || !aligned(p.fac, 32) || !aligned(scratch, 32)) return cudaErrorInvalidValue;
  p.d = d;
  for (int i = 0; i < d.ndir; i++) {
    if (!aligned(w_hh[i], 16)) return cudaErrorInvalidValue;
    p.w_hh[i] = w_hh[i];
  }
  char* w = (char*)scratch;
  p.sync = (uint32_t*)w;
  p.ring = (uint32_t*)(w + kSyncBytes);
  p.status = status;
  p.timeout_ns = (unsigned long long)(timeout_s * 1e9);
  p.prof = g_prof;
  return cudaSuccess;
}

}  // namespace

void gru_persistent_set_profile(unsigned long long* stamps) { g_prof = stamps; }

bool gru_persistent_supported(const GruDims& d, int device) {
  if (!dims_ok(d)) return false;
  int major = 0, sms = 0, smem_optin = 0;
  if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device) != cudaSuccess || major != 10) return false;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return false;
  if (cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess) return false;
  return smem_optin >= 227 * 1024 && d.H / kUnits * d.ndir <= sms;
}

size_t gru_persistent_workspace_bytes(const GruDims& d) { return dims_ok(d) ? exchange_bytes(d) : 0; }

// Behind the ring every block has two slots of partial sums, three per 16 bytes, from every member of its group (its own stay in shared
// memory; their place is not used).
size_t gru_persistent_scratch_bytes(const GruDims& d) {
  if (!dims_ok(d)) return 0;
  return kSyncBytes + ring_bytes(d) + (size_t)d.ndir * (d.H / kUnits) * 2 * ((d.B + 2) / 3) * exchange_rows(d) * 16;
}

cudaError_t gru_persistent_forward(const GruDims& d, const float* const* w_hh, const float* const* b_hh, const float* gx, float* y,
                                   float* rsv, float* fac, void* scratch, uint32_t* status, double timeout_s, cudaStream_t stream) {
  Params p{};
  p.rsv = (float4*)rsv;
  p.fac = fac;
  const cudaError_t e = start(p, d, w_hh, scratch, status, timeout_s);
  if (e != cudaSuccess) return e;
  for (int i = 0; i < d.ndir; i++) p.b_hh[i] = b_hh[i];
  p.gx = gx;
  p.y = y;
  return launch_forward(p, stream);
}

cudaError_t gru_persistent_backward(const GruDims& d, const float* const* w_hh, const float* y, const float* rsv, const float* fac, const float* dy,
                                    float* dg, float* db, void* scratch, uint32_t* status, double timeout_s, cudaStream_t stream) {
  Params p{};
  p.rsv = (float4*)const_cast<float*>(rsv);
  p.fac = const_cast<float*>(fac);
  const cudaError_t e = start(p, d, w_hh, scratch, status, timeout_s);
  if (e != cudaSuccess) return e;
  p.y = const_cast<float*>(y);
  p.dy = dy;
  p.dg = dg;
  p.db = db;
  return launch_backward(p, stream);
}

}  // namespace gpu
}  // namespace bc

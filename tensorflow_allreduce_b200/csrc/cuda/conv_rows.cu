// Row convolutions on tcgen05 (see conv_rows.h).
//
// The operands are brought into shared memory by ordinary loads that transpose NCHW on the way, so no layout conversion
// touches memory: cuDNN's kernels for these shapes spent 0.7 ms per training step on that, and ran at 10 to 30 % of
// the TF32 rate because 32 output channels fill a quarter of an MMA tile.
//
// Forward and input gradient (rows_kernel). 32 channels are one 128-byte row of the operand layout. A block makes R output
// rows of one image over up to 384 columns. For an input row i (its pixels are the M side, 128 per MMA, K = its 32
// channels) the N side stacks the weights of the R output rows that i contributes to: 32 R rows, which lie one
// behind the other in a packed copy of the weights, so MMAs are N = 160 to 256 wide instead of 32. The horizontal taps move
// the start of the pixel operand by one 128-byte row each; the row is loaded once for all of them. Accumulators of all R rows
// stay in tensor memory until the end.
//   conv 1 (one input channel, stride 2 x 2) is the same with pairs of input rows as rows and (row of the pair, horizontal
//   tap) as the 32 channels, without taps of its own.
//
// Weight gradient (wgrad_kernel). K is the image column, as NCHW has it. M = 128 rows: horizontal shift x input channel (conv 1:
// 8 input rows x 16 shifts), N = the output rows that an input row meets, 32 channels each, held in a ring
// of rows in shared memory as the input row advances. Every block adds up a share of images and column chunks of 32 and
// writes its partial sums; a second kernel adds the blocks' partial sums in fixed order.
//
// Every wait is bounded and ends in the status word.
#include "conv_rows.h"

#include <algorithm>

#include "tcgen05_prims.cuh"

namespace bc {
namespace gpu {

namespace {

using namespace tc;

constexpr uint32_t kConvTimeout = 8u;
constexpr int kCo = 32;                      // output channels, and the "channels" of an operand row
constexpr int kRow = 128;                    // bytes of one
constexpr int kMaxCols = 384;                // output columns of a block of rows_kernel
constexpr uint32_t kTmem = 512;

enum Mode { FORWARD = 0, DGRAD = 1, GATHER = 2 };   // GATHER: forward with one input channel

__device__ __forceinline__ void st_smem16(uint32_t at, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// ---- forward and input gradient ------------------------------------------------------------------

struct RowsParams {
  const float* x;
  float* y;
  const char* w;             // packed weights: [tap][parity][table row][32 n][32 k], swizzled
  int Hi, Wi, Ho, Wo;        // of the tensors that this pass reads and writes
  int KH, ph, pad;           // vertical kernel size and padding, horizontal offset of the operand row
  int taps, R, T;            // horizontal taps; output rows and 128-column tiles of a block
  int table;                 // rows of 32 in one table
  uint32_t* status;
  unsigned long long timeout_ns;
};

// Weight tables. FORWARD / GATHER: entry t holds m = mhi - t (kernel row 2 m + parity, or pair of rows m); DGRAD: kernel row t - (R - 1).
// Entries outside the kernel are zero; the block at table row `start` has the weights of output row r at start + r.
__host__ __device__ inline int half_taps(int KH) { return (KH + 1) / 2; }
__host__ __device__ inline int table_rows(int mode, int KH, int R) { return (mode == DGRAD ? KH : half_taps(KH)) + 2 * (R - 1); }

constexpr int kPackThreads = 256;
// One 16-byte chunk of the packed weights per thread.
template <int MODE>
__global__ void __launch_bounds__(kPackThreads) pack_kernel(const float* __restrict__ w, uint4* __restrict__ out, int KH, int KW, int R, int table, int total) {
  const int idx = blockIdx.x * kPackThreads + threadIdx.x;
  if (idx >= total) return;
  const int chunk = idx & 7, n = (idx >> 3) & 31, tt = idx >> 8;
  const int t = tt % table, tp = tt / table;
  constexpr int kPar = MODE == FORWARD ? 2 : 1;
  const int par = tp % kPar, tap = tp / kPar;
  uint32_t v[4];
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const int k = chunk * 4 + e;
    float f = 0.f;
    if (MODE == FORWARD) {
      const int kh = 2 * (half_taps(KH) - 1 + R - 1 - t) + par;
      if (kh >= 0 && kh < KH) f = w[((n * kCo + k) * KH + kh) * KW + tap];
    } else if (MODE == DGRAD) {
      const int kh = t - (R - 1);
      if (kh >= 0 && kh < KH) f = w[((k * kCo + n) * KH + kh) * KW + (KW - 1 - tap)];
    } else {
      const int kh = 2 * (half_taps(KH) - 1 + R - 1 - t) + (k >> 4), kw = k & 15;
      if (kh >= 0 && kh < KH && kw < KW) f = w[(n * KH + kh) * KW + kw];
    }
    v[e] = to_tf32(f);
  }
  out[(idx & ~7) + (chunk ^ (n & 7))] = make_uint4(v[0], v[1], v[2], v[3]);
}

constexpr int kLoaders = 256;                // eight warps, one per 16-byte chunk (four channels) of the operand rows
constexpr int kRowsThreads = kLoaders + 64;  // + a warp for the MMAs + a warp for the weights
constexpr int kBStages = 4;
__host__ __device__ inline int a_rows(int T) { return T * 128 + 16; }
inline int rows_smem(int R, int T) { return 1024 + 2 * a_rows(T) * kRow + kBStages * R * kCo * kRow + 256; }

template <int MODE>
__global__ void __launch_bounds__(kRowsThreads, 1) rows_kernel(const __grid_constant__ RowsParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n = blockIdx.x, o0 = blockIdx.y * p.R, w0 = blockIdx.z * kMaxCols;
  const int R = p.R, T = p.T, taps = MODE == GATHER ? 1 : p.taps;
  const int a_bytes = a_rows(T) * kRow, b_bytes = R * kCo * kRow;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 2 * a_bytes + kBStages * b_bytes);   // a full[2], a empty[2], b full, b empty, done
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 5 + 2 * kBStages);
  volatile int* abort_s = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t a_full = smem_u32(bars), a_empty = a_full + 16, b_full = a_full + 32, b_empty = b_full + 8 * kBStages, done = b_empty + 8 * kBStages;
  const uint32_t a_addr = smem_u32(smem), b_addr = a_addr + 2 * a_bytes;
  if (tid == 0) {
    for (int i = 0; i < 2; i++) { mbar_init(a_full + 8 * i, kLoaders / 32); mbar_init(a_empty + 8 * i, 1); }
    for (int i = 0; i < kBStages; i++) { mbar_init(b_full + 8 * i, 1); mbar_init(b_empty + 8 * i, 1); }
    mbar_init(done, 1);
    *abort_s = 0;
    mbar_init_fence();
  }
  if (warp == kLoaders / 32) tmem_alloc(tmem_slot, kTmem);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // Input rows (GATHER: pairs of rows) that meet the block's output rows, and the table row of the weights for one of them.
  int lo, hi;
  if (MODE == FORWARD) {
    lo = 2 * o0 - p.ph;
    hi = 2 * (o0 + R - 1) - p.ph + p.KH - 1;
  } else if (MODE == DGRAD) {
    lo = (o0 + p.ph - p.KH + 2) >> 1;
    hi = (o0 + R - 1 + p.ph) >> 1;
  } else {
    lo = o0 - p.ph / 2;
    hi = o0 + R - 1 - p.ph / 2 + half_taps(p.KH) - 1;
  }
  lo = max(lo, 0);
  hi = min(hi, (MODE == GATHER ? (p.Hi + 1) / 2 : p.Hi) - 1);
  const int mhi = half_taps(p.KH) - 1 + R - 1;
  auto table_at = [&](int i, int tap) -> size_t {     // in rows of 32 x 128 bytes
    if (MODE == FORWARD) {
      const int q = i + p.ph - 2 * o0;
      return (size_t)(tap * 2 + (q & 1)) * p.table + (mhi - (q >> 1));
    } else if (MODE == DGRAD) {
      return (size_t)tap * p.table + (o0 + p.ph - 2 * i + R - 1);
    }
    return (size_t)(mhi - (i - o0 + p.ph / 2));
  };

  bool ok = true;
  if (warp < kLoaders / 32) {
    // ---------------- loaders: pixel rows of 32 channels ----------------
    const int chunk = warp;
    const int cols = T * 128 + taps - 1;
    const size_t plane = (size_t)p.Hi * p.Wi;
    const float* xn = p.x + (size_t)n * (MODE == GATHER ? 1 : kCo) * plane;
    for (int i = lo, k = 0; i <= hi; i++, k++) {
      const int st = k & 1;
      if (k >= 2) ok = ok && mbar_wait(a_empty + 8 * st, (uint32_t)((k >> 1) - 1) & 1, p.timeout_ns, abort_s);
      const uint32_t dst = a_addr + st * a_bytes;
      for (int px0 = 0; px0 < cols; px0 += 128) {
        float v[4][4];
        if (MODE == GATHER) {
          const int h = 2 * i + (chunk >> 2), t0 = (chunk & 3) * 4;
          const float* row = xn + (size_t)h * p.Wi;
#pragma unroll
          for (int u = 0; u < 4; u++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
              const int col = 2 * (w0 + px0 + u * 32 + lane) + t0 + e - p.pad;
              v[u][e] = (h < p.Hi && col >= 0 && col < p.Wi && t0 + e < p.taps) ? __ldg(row + col) : 0.f;
            }
        } else {
          const float* row = xn + (size_t)(4 * chunk) * plane + (size_t)i * p.Wi;
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const int col = w0 + px0 + u * 32 + lane - p.pad;
            const bool in = col >= 0 && col < p.Wi;
#pragma unroll
            for (int e = 0; e < 4; e++) v[u][e] = in ? __ldg(row + e * plane + col) : 0.f;
          }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int px = px0 + u * 32 + lane;
          if (px < cols)
            st_smem16(dst + px * kRow + ((chunk ^ (px & 7)) << 4), to_tf32(v[u][0]), to_tf32(v[u][1]), to_tf32(v[u][2]), to_tf32(v[u][3]));
        }
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(a_full + 8 * st);
    }
    ok = ok && mbar_wait(done, 0, 4 * p.timeout_ns, abort_s);
    ok = __all_sync(0xffffffffu, ok) != 0;
    tc_fence_after();
    if (ok) {
      const int quarter = warp & 3;
      const size_t oplane = (size_t)p.Ho * p.Wo;
      for (int u = warp >> 2; u < T * R; u += 2) {
        const int t = u / R, r = u % R;
        uint32_t v[32];
        tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(u * 32), v);
        const int col = w0 + t * 128 + quarter * 32 + lane;
        if (o0 + r < p.Ho && col < p.Wo) {
          float* o = p.y + (size_t)n * kCo * oplane + (size_t)(o0 + r) * p.Wo + col;
#pragma unroll
          for (int c = 0; c < 32; c++) o[c * oplane] = __uint_as_float(v[c]);
        }
      }
      tc_fence_before();
    }
  } else if (warp == kLoaders / 32) {
    // ---------------- MMAs ----------------
    const bool leader = elect_one();
    const uint32_t idesc = idesc_tf32(128, R * kCo);
    const uint64_t a_desc = operand_desc(a_addr), b_desc = operand_desc(b_addr);
    uint32_t acc = 0;
    int b = 0;
    for (int i = lo, k = 0; ok && i <= hi; i++, k++) {
      const int st = k & 1;
      ok = mbar_wait(a_full + 8 * st, (uint32_t)(k >> 1) & 1, p.timeout_ns, abort_s);
      for (int tap = 0; tap < taps; tap++, b++) {
        const int bs = b % kBStages;
        ok = ok && mbar_wait(b_full + 8 * bs, (uint32_t)(b / kBStages) & 1, p.timeout_ns, abort_s);
        ok = __all_sync(0xffffffffu, ok) != 0;
        if (!ok) break;
        tc_fence_after();
        if (leader) {
          const uint64_t bd = b_desc + (uint64_t)(bs * b_bytes >> 4);
          for (int t = 0; t < T; t++) {
            const uint64_t ad = a_desc + (uint64_t)((st * a_bytes + (t * 128 + tap) * kRow) >> 4);
#pragma unroll
            for (int ks = 0; ks < 4; ks++) tc_mma_ss(tmem + t * R * kCo, ad + 2 * ks, bd + 2 * ks, idesc, ks ? 1u : acc);
          }
          tc_commit(b_empty + 8 * bs);
          if (tap == taps - 1) tc_commit(a_empty + 8 * st);
        }
        acc = 1;
        __syncwarp();
      }
    }
    if (leader) tc_commit(done);      // also the end of whatever is in flight when a wait has run out
    __syncwarp();
    ok = mbar_wait(done, 0, p.timeout_ns, nullptr) && ok;
  } else {
    // ---------------- weights ----------------
    if (elect_one()) {
      int b = 0;
      for (int i = lo; ok && i <= hi; i++)
        for (int tap = 0; ok && tap < taps; tap++) {
          const int bs = b % kBStages;
          if (b >= kBStages) ok = mbar_wait(b_empty + 8 * bs, (uint32_t)(b / kBStages - 1) & 1, p.timeout_ns, abort_s);
          if (!ok) break;
          mbar_expect_tx(b_full + 8 * bs, (uint32_t)b_bytes);
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                       ::"r"(b_addr + bs * b_bytes), "l"(p.w + table_at(i, tap) * (kCo * kRow)), "r"((uint32_t)b_bytes), "r"(b_full + 8 * bs) : "memory");
          b++;
        }
      // No copy may be in flight when the block ends: the MMA warp has waited for all of them unless it gave up.
      for (int back = min(b, kBStages); back > 0; back--)
        mbar_wait(b_full + 8 * ((b - back) % kBStages), (uint32_t)((b - back) / kBStages) & 1, p.timeout_ns, nullptr);
    }
    __syncwarp();
  }
  if (!ok) {
    *abort_s = 1;
    atomicOr(p.status, kConvTimeout);
  }
  __syncthreads();
  if (warp == kLoaders / 32) tmem_free(tmem, kTmem);
}


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
// Every wait is bounded and ends in the status word; a block that gives up waits for its own copies and MMAs before it ends.
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
        if (lo > hi) {             // no input row meets these output rows (trailing rows of an input gradient)
#pragma unroll
          for (int c = 0; c < 32; c++) v[c] = 0u;
        }
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
    ok = mbar_drain(done, 0) && ok;
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
        mbar_drain(b_full + 8 * ((b - back) % kBStages), (uint32_t)((b - back) / kBStages) & 1);
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

// ---- weight gradient -------------------------------------------------------------------------------

// HB input rows of one parity at a time. HB = 1: 32 input channels, four horizontal shifts, M row = shift * 32 + channel.
// HB = 8: one input channel, 16 shifts, M row = (input row) * 16 + shift. Kernel row kh = 2 m + parity; an input row block at
// h, with e = (h + ph - parity) / 2, meets output row oh = e - m' where m' = m - (row of the block).
template <int HB> struct WgradShape {
  static constexpr int kCi = HB == 1 ? 32 : 1;
  static constexpr int kAStages = HB == 1 ? 4 : 2, kRing = HB == 1 ? 16 : 32;
  static constexpr int smem = 1024 + kAStages * 128 * kRow + kRing * kCo * kRow + 256;
};
constexpr int kMaxM = 16;                    // values of m' per block: 512 columns of tensor memory
constexpr int kGroup = 256;                  // threads of one of the two loader groups, which take every other step
constexpr int kWgradThreads = 2 * kGroup + 32;

struct WgradParams {
  const float* x;
  const float* dy;
  float* part;               // [block][128 rows][kMaxM][32]
  int N, Hi, Wi, Ho, Wo, KH, KW, ph, pw;
  int kinds, per_kind;       // block b works on kind b % kinds
  uint32_t* status;
  unsigned long long timeout_ns;
};

// Kind: parity of the kernel row, and HB = 1: which four shifts; HB = 8: which half of the values of m'.
struct Kind { int par, j, mb, mc; };
template <int HB>
__host__ __device__ inline Kind kind_of(int kind, int KH) {
  Kind k;
  k.par = kind & 1;
  const int m = (KH - k.par + 1) / 2, all = m + HB - 1;
  if (HB == 1) {
    k.j = kind >> 1;
    k.mb = 0;
    k.mc = m;
  } else {
    const int first = (all + 1) / 2;
    k.j = 0;
    k.mb = -(HB - 1) + ((kind >> 1) ? first : 0);
    k.mc = (kind >> 1) ? all - first : first;
  }
  return k;
}

template <int HB>
__global__ void __launch_bounds__(kWgradThreads, 1) wgrad_kernel(const __grid_constant__ WgradParams p) {
  using S = WgradShape<HB>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const Kind kd = kind_of<HB>(blockIdx.x % p.kinds, p.KH);
  const int first_unit = blockIdx.x / p.kinds;
  const uint32_t a_addr = smem_u32(smem), r_addr = a_addr + S::kAStages * 128 * kRow;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::kAStages * 128 * kRow + S::kRing * kCo * kRow);    // full, empty, done
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S::kAStages + 1);
  volatile int* abort_s = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t full = smem_u32(bars), empty = full + 8 * S::kAStages, done = empty + 8 * S::kAStages;
  if (tid == 0) {
    for (int i = 0; i < S::kAStages; i++) { mbar_init(full + 8 * i, kGroup / 32); mbar_init(empty + 8 * i, 1); }
    mbar_init(done, 1);
    *abort_s = 0;
    mbar_init_fence();
  }
  if (warp == kWgradThreads / 32 - 1) tmem_alloc(tmem_slot, kTmem);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (warp < 4) {
    float z[16];
#pragma unroll
    for (int i = 0; i < 16; i++) z[i] = 0.f;
    for (int c = 0; c < (int)kTmem; c += 16) tmem_st16(tmem + ((uint32_t)(warp * 32) << 16) + c, z);
    tmem_st_wait();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  // A unit is one image and 32 output columns; its steps go down the input rows of the parity.
  const int chunks = (p.Wo + 31) / 32, units = p.N * chunks;
  const int h0 = (kd.par + p.ph) & 1, steps = (p.Hi - h0 + 2 * HB - 1) / (2 * HB), e0 = (h0 + p.ph - kd.par) / 2;
  auto slot_of = [](int oh) { return (uint32_t)(-oh) & (S::kRing - 1); };

  bool ok = true;
  if (warp < 2 * kGroup / 32) {
    // ---------------- loaders ----------------
    const int group = tid / kGroup, t = tid % kGroup, chunk = t & 7, tr = t >> 3;      // tr: row of 32 within a batch of 256 chunks
    const size_t xplane = (size_t)p.Hi * p.Wi, yplane = (size_t)p.Ho * p.Wo;
    int step0 = 0;                                             // number of the unit's first step
    for (int u = first_unit; u < units; u += p.per_kind, step0 += steps) {
      const int n = u / chunks, w0 = (u % chunks) * 32;
      const float* xn = p.x + (size_t)n * S::kCi * xplane;
      const float* yn = p.dy + (size_t)n * kCo * yplane + (size_t)tr * yplane + w0 + 4 * chunk;
      for (int k = (step0 + group) & 1; k < steps; k += 2) {
        const int s = step0 + k, st = s % S::kAStages, h = h0 + 2 * HB * k, e = e0 + HB * k;
        // A operand: HB = 1: seven columns make the chunk of four shifts; HB = 8: four rows of the operand, one chunk each
        float f[16];
        if (HB == 1) {
          const int col = w0 + 4 * chunk + 4 * kd.j - p.pw;
          const float* row = xn + (size_t)tr * xplane + (size_t)h * p.Wi;
#pragma unroll
          for (int i = 0; i < 7; i++) f[i] = (col + i >= 0 && col + i < p.Wi) ? __ldg(row + col + i) : 0.f;
        } else {
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const int r = tr + 32 * i, hh = h + 2 * (r >> 4), sh = r & 15;
#pragma unroll
            for (int c = 0; c < 4; c++) {
              const int col = 2 * (w0 + 4 * chunk + c) + sh - p.pw;
              f[4 * i + c] = (hh < p.Hi && sh < p.KW && col >= 0 && col < p.Wi) ? __ldg(xn + (size_t)hh * p.Wi + col) : 0.f;
            }
          }
        }
        // rows of dy that this step adds to the ring, [lo, hi]: HB of them, all that its window holds at the first step of a unit
        const int hi = min(e - kd.mb, p.Ho - 1), lo = max(k == 0 ? e - kd.mb - kd.mc + 1 : e - kd.mb - HB + 1, 0);
        constexpr int kBatch = HB == 1 ? 1 : 4;
        float g[kBatch][4];
        auto load_rows = [&](int from) {
#pragma unroll
          for (int b = 0; b < kBatch; b++)
#pragma unroll
            for (int c = 0; c < 4; c++)
              g[b][c] = (from + b <= hi && w0 + 4 * chunk + c < p.Wo) ? __ldg(yn + (size_t)(from + b) * p.Wo + c) : 0.f;
        };
        load_rows(lo);
        // The stage is free when the MMAs of kAStages steps ago are done; so is then the ring row that is overwritten
        // (kRing > (kAStages - 1) HB + mc - 1). At the start of a unit the window jumps: wait for all steps before it.
        if (s >= S::kAStages) ok = ok && mbar_wait(empty + 8 * st, (uint32_t)(s / S::kAStages - 1) & 1, p.timeout_ns, abort_s);
        if (k < S::kAStages && step0 > 0) ok = ok && mbar_wait(empty + 8 * ((step0 - 1) % S::kAStages), (uint32_t)((step0 - 1) / S::kAStages) & 1, p.timeout_ns, abort_s);
        const uint32_t dst = a_addr + st * (128 * kRow), sw = (uint32_t)((chunk ^ (tr & 7)) << 4);
        if (HB == 1) {
          uint32_t q[7];
#pragma unroll
          for (int i = 0; i < 7; i++) q[i] = to_tf32(f[i]);
#pragma unroll
          for (int i = 0; i < 4; i++) st_smem16(dst + (i * 32 + tr) * kRow + sw, q[i], q[i + 1], q[i + 2], q[i + 3]);
        } else {
#pragma unroll
          for (int i = 0; i < 4; i++)
            st_smem16(dst + (i * 32 + tr) * kRow + sw, to_tf32(f[4 * i]), to_tf32(f[4 * i + 1]), to_tf32(f[4 * i + 2]), to_tf32(f[4 * i + 3]));
        }
        for (int oh = lo; oh <= hi; oh += kBatch) {
#pragma unroll
          for (int b = 0; b < kBatch; b++)
            if (oh + b <= hi)
              st_smem16(r_addr + slot_of(oh + b) * (kCo * kRow) + tr * kRow + sw, to_tf32(g[b][0]), to_tf32(g[b][1]), to_tf32(g[b][2]), to_tf32(g[b][3]));
          if (oh + kBatch <= hi) load_rows(oh + kBatch);
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(full + 8 * st);
      }
    }
    ok = ok && mbar_wait(done, 0, 4 * p.timeout_ns, abort_s);
    ok = __all_sync(0xffffffffu, ok) != 0;
    tc_fence_after();
    if (ok) {
      const int quarter = warp & 3;
      float* out = p.part + ((size_t)blockIdx.x * 128 + quarter * 32 + lane) * (kMaxM * kCo);
      for (int mi = warp >> 2; mi < kd.mc; mi += 2 * kGroup / 128) {
        uint32_t v[32];
        tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(mi * kCo), v);
#pragma unroll
        for (int c = 0; c < 8; c++) *reinterpret_cast<uint4*>(out + mi * kCo + 4 * c) = make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
      }
      tc_fence_before();
    }
  } else {
    // ---------------- MMAs ----------------
    const bool leader = elect_one();
    const uint64_t a_desc = operand_desc(a_addr), b_desc = operand_desc(r_addr);
    int s = 0;
    for (int u = first_unit; ok && u < units; u += p.per_kind) {
      for (int k = 0; k < steps; k++, s++) {
        const int st = s % S::kAStages, e = e0 + HB * k;
        ok = mbar_wait(full + 8 * st, (uint32_t)(s / S::kAStages) & 1, p.timeout_ns, abort_s);
        ok = __all_sync(0xffffffffu, ok) != 0;
        if (!ok) break;
        tc_fence_after();
        if (leader) {
          const uint64_t ad = a_desc + (uint64_t)(st * (128 * kRow) >> 4);
          // values of m' whose output row exists; their ring slots ascend with m' and may wrap once
          const int m_end = min(kd.mb + kd.mc, e + 1);
          for (int m = max(kd.mb, e - p.Ho + 1); m < m_end;) {
            const uint32_t slot = slot_of(e - m);
            const int len = min(min(m_end - m, S::kRing - (int)slot), 8);
            const uint64_t bd = b_desc + (uint64_t)(slot * (kCo * kRow) >> 4);
            const uint32_t idesc = idesc_tf32(128, len * kCo), d = tmem + (uint32_t)((m - kd.mb) * kCo);
#pragma unroll
            for (int ks = 0; ks < 4; ks++) tc_mma_ss(d, ad + 2 * ks, bd + 2 * ks, idesc, 1u);
            m += len;
          }
          tc_commit(empty + 8 * st);
        }
        __syncwarp();
      }
    }
    if (leader) tc_commit(done);
    __syncwarp();
    ok = mbar_drain(done, 0) && ok;
  }
  if (!ok) {
    *abort_s = 1;
    atomicOr(p.status, kConvTimeout);
  }
  __syncthreads();
  if (warp == kWgradThreads / 32 - 1) tmem_free(tmem, kTmem);
}

// dw[co][ci][kh][kw]: sum over the blocks of its kind (and, HB = 8, over the input rows of a block step). One block per
// (ci, kh, kw), thread (co, y): y takes every eighth block, or input row y.
template <int HB>
__global__ void __launch_bounds__(256) wgrad_sum_kernel(const float* __restrict__ part, float* __restrict__ dw, int KH, int KW, int kinds, int per_kind) {
  using S = WgradShape<HB>;
  const int co = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int kw = blockIdx.x % KW, kh = blockIdx.x / KW % KH, ci = blockIdx.x / (KW * KH);
  int kind = kh & 1, row, mp = kh >> 1;
  if (HB == 1) {
    kind += 2 * (kw >> 2);
    row = (kw & 3) * 32 + ci;
  } else {
    mp -= y;
    row = y * 16 + kw;
    if (mp >= kind_of<HB>(kind + 2, KH).mb) kind += 2;
  }
  const int mi = mp - kind_of<HB>(kind, KH).mb;
  float v = 0.f;
  const size_t block = (size_t)128 * kMaxM * kCo;
  const float* src = part + (size_t)row * (kMaxM * kCo) + mi * kCo + co;
#pragma unroll 4
  for (int i = HB == 1 ? y : 0; i < per_kind; i += HB == 1 ? 8 : 1) v += __ldg(src + (size_t)(kind + kinds * i) * block);
  __shared__ float sum[8][32];
  sum[y][co] = v;
  __syncthreads();
  if (y == 0) {
#pragma unroll
    for (int i = 1; i < 8; i++) v += sum[i][co];
    dw[(((size_t)co * S::kCi + ci) * KH + kh) * KW + kw] = v;
  }
}

// ---- host side -------------------------------------------------------------------------------------

int tiles_of(int cols) { return std::min((cols + 127) / 128, kMaxCols / 128); }
int sm_count() {
  int dev = 0, n = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

// Output rows per block, at most what tensor memory holds (16 units of 32 columns over all tiles) and N = 256 per MMA. More
// rows share an input row's loads and make wider MMAs, but also compute more rows than the kernel is high and leave fewer
// blocks: the number that needs the fewest cycles in the fullest SM. An MMA measured 110 cycles up to 5 rows, 17 per row above; conv 1
// is bound by its loads, 1340 cycles per row and tile. (32 -> 32 channels, 81 x 50, 4 images: 5 blocks of 8 rows 156 us, chosen rows
// 93 us; 32 images of 81 x 350 stay at 5 rows: 470 us, with 4 rows for the input gradient 466 instead of 393 us.)
int rows_of(int mode, const ConvDims& d, int Ho, int Wo, int sms) {
  const int T = tiles_of(Wo);
  int best = 1;
  double least = 0;
  for (int R = 1; R <= std::min(16 / T, 8); R++) {
    const int rows = mode == FORWARD ? d.KH + 2 * (R - 1) : mode == DGRAD ? (d.KH + R) / 2 : half_taps(d.KH) + R - 1;
    const long blocks = (long)d.N * ((Ho + R - 1) / R) * ((Wo + kMaxCols - 1) / kMaxCols);
    const double row = mode == GATHER ? std::max(1340, 4 * 17 * R) : d.KW * 4 * std::max(110, 17 * R);
    const double cycles = (double)((blocks + sms - 1) / sms) * (5000 + rows * row * T);
    if (R == 1 || cycles < least) {
      least = cycles;
      best = R;
    }
  }
  return best;
}

size_t table_bytes(int mode, const ConvDims& d, int R) {
  const int tables = mode == GATHER ? 1 : d.KW * (mode == FORWARD ? 2 : 1);
  return (size_t)tables * table_rows(mode, d.KH, R) * kCo * kRow;
}

template <int HB> int wgrad_kinds(const ConvDims& d) { return 2 * (HB == 1 ? (d.KW + 3) / 4 : 2); }
template <int HB> int wgrad_per_kind(const ConvDims& d) {
  const int units = d.N * ((d.Wo() + 31) / 32);
  return std::max(1, std::min(std::min(sm_count(), 256) / wgrad_kinds<HB>(d), units));
}

template <typename K>
cudaError_t allow_smem(K kernel) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
}

template <int MODE>
cudaError_t run_rows(const ConvDims& d, const float* x, const float* w, float* y, int Hi, int Wi, int Ho, int Wo, int pad, void* scratch,
                     uint32_t* status, double timeout_s, cudaStream_t stream) {
  RowsParams p;
  p.T = tiles_of(Wo);
  p.R = rows_of(MODE, d, Ho, Wo, sm_count());
  p.x = x;
  p.y = y;
  p.w = (const char*)scratch;
  p.Hi = Hi; p.Wi = Wi; p.Ho = Ho; p.Wo = Wo;
  p.KH = d.KH; p.ph = d.ph; p.pad = pad;
  p.taps = d.KW;
  p.table = table_rows(MODE, d.KH, p.R);
  p.status = status;
  p.timeout_ns = (unsigned long long)(timeout_s * 1e9);
  const int total = (int)(table_bytes(MODE, d, p.R) / 16);
  pack_kernel<MODE><<<(total + kPackThreads - 1) / kPackThreads, kPackThreads, 0, stream>>>(w, (uint4*)scratch, d.KH, d.KW, p.R, p.table, total);
  cudaError_t e = allow_smem(rows_kernel<MODE>);
  if (e != cudaSuccess) return e;
  const dim3 grid(d.N, (Ho + p.R - 1) / p.R, (Wo + kMaxCols - 1) / kMaxCols);
  // at least more than half of an SM's shared memory: a block takes all of tensor memory
  rows_kernel<MODE><<<grid, kRowsThreads, std::max(rows_smem(p.R, p.T), 120 * 1024), stream>>>(p);
  return cudaGetLastError();
}

template <int HB>
cudaError_t run_wgrad(const ConvDims& d, const float* x, const float* dy, float* dw, void* scratch, uint32_t* status, double timeout_s, cudaStream_t stream) {
  WgradParams p;
  p.x = x;
  p.dy = dy;
  p.part = (float*)scratch;
  p.N = d.N; p.Hi = d.H; p.Wi = d.W; p.Ho = d.Ho(); p.Wo = d.Wo(); p.KH = d.KH; p.KW = d.KW; p.ph = d.ph; p.pw = d.pw;
  p.kinds = wgrad_kinds<HB>(d);
  p.per_kind = wgrad_per_kind<HB>(d);
  p.status = status;
  p.timeout_ns = (unsigned long long)(timeout_s * 1e9);
  cudaError_t e = allow_smem(wgrad_kernel<HB>);
  if (e != cudaSuccess) return e;
  wgrad_kernel<HB><<<p.kinds * p.per_kind, kWgradThreads, WgradShape<HB>::smem, stream>>>(p);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  wgrad_sum_kernel<HB><<<d.Cin * d.KH * d.KW, 256, 0, stream>>>(p.part, dw, d.KH, d.KW, p.kinds, p.per_kind);
  return cudaGetLastError();
}

bool dims_ok(const ConvDims& d) {
  if (d.N < 1 || d.N > 65535 || d.H < 1 || d.W < 1 || d.KH < 1 || d.KW < 1 || d.KW > 16 || d.ph < 0 || d.pw < 0 || d.ph >= d.KH || d.pw >= d.KW) return false;
  if (d.H + 2 * d.ph < d.KH || d.W + 2 * d.pw < d.KW || d.H > 4096 || d.W > (1 << 20)) return false;
  if (d.Cin == 32) return d.stride_w == 1 && (d.KH + 1) / 2 <= 13;                   // the ring of the weight gradient holds its window
  return d.Cin == 1 && d.stride_w == 2 && d.ph % 2 == 0 && (d.KH + 1) / 2 + 7 <= 2 * kMaxM;
}

}  // namespace

bool conv_rows_supported(const ConvDims& d, int device) {
  if (!dims_ok(d)) return false;
  int major = 0;
  return cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device) == cudaSuccess && major == 10;
}

size_t conv_rows_scratch_bytes(const ConvDims& d) {
  if (!dims_ok(d)) return 0;
  const size_t block = (size_t)128 * kMaxM * kCo * 4;
  if (d.Cin == 1) return std::max(table_bytes(GATHER, d, 8), block * wgrad_kinds<8>(d) * wgrad_per_kind<8>(d));
  return std::max(std::max(table_bytes(FORWARD, d, 8), table_bytes(DGRAD, d, 8)), block * wgrad_kinds<1>(d) * wgrad_per_kind<1>(d));
}

cudaError_t conv_rows_forward(const ConvDims& d, const float* x, const float* w, float* y, void* scratch, uint32_t* status, double timeout_s,
                              cudaStream_t stream) {
  if (!dims_ok(d)) return cudaErrorInvalidValue;
  if (d.Cin == 1) return run_rows<GATHER>(d, x, w, y, d.H, d.W, d.Ho(), d.Wo(), d.pw, scratch, status, timeout_s, stream);
  return run_rows<FORWARD>(d, x, w, y, d.H, d.W, d.Ho(), d.Wo(), d.pw, scratch, status, timeout_s, stream);
}

cudaError_t conv_rows_backward_input(const ConvDims& d, const float* dy, const float* w, float* dx, void* scratch, uint32_t* status,
                                     double timeout_s, cudaStream_t stream) {
  if (!dims_ok(d) || d.Cin != 32) return cudaErrorInvalidValue;
  return run_rows<DGRAD>(d, dy, w, dx, d.Ho(), d.Wo(), d.H, d.W, d.KW - 1 - d.pw, scratch, status, timeout_s, stream);
}

cudaError_t conv_rows_backward_weight(const ConvDims& d, const float* x, const float* dy, float* dw, void* scratch, uint32_t* status,
                                      double timeout_s, cudaStream_t stream) {
  if (!dims_ok(d)) return cudaErrorInvalidValue;
  return d.Cin == 1 ? run_wgrad<8>(d, x, dy, dw, scratch, status, timeout_s, stream) : run_wgrad<1>(d, x, dy, dw, scratch, status, timeout_s, stream);
}

}  // namespace gpu
}  // namespace bc

// Forward pass of the persistent GRU layer for sm_100a (see gru_persistent.h for the interface).
//
// Work split. Direction d of a layer is run by H/16 blocks (grid.y = direction); block c owns the hidden units [16c, 16c+16), keeps the 48
// weight rows of their gates on chip for the whole sequence and multiplies them with ALL of h_{t-1}, so that a step has one
// exchange between blocks: the new h. Each time step a block
//   1. polls h_{t-1} in a ring in global memory and puts it into shared memory in the 128-byte swizzle,
//   2. multiplies with tcgen05.mma: the weights are the M side and live in tensor memory, the batch is the N side, K = 16 per instruction,
//   3. reads the accumulator back, applies the gates, and puts its part of h_t into the ring.
//
// Operands. Weights are split into two fp16 values, w = (hi + lo) / scale, that are two ROWS of the M side: 96 of 128 rows in use, one
// instruction for both. The scale is a power of two per row that puts the row's largest weight between 2^14 and 2^15. h_{t-1}, which is at
// most 1 in magnitude (the initial state is zero), is multiplied by 2^15 and rounded to fp16 with nine explicit bits of mantissa; the
// tenth belongs to the exchange. Products of fp16 values are exact and sums fp32. Against TF32 operands, whose weights and h
// the tensor core cuts to ten bits, towards zero, the error of h has the same mean square and no bias, and the weights have 22 bits.
// What it buys: 2 bytes of operand per value instead of 4, and K = 16 instead of 8 at the same cost per instruction (16 cycles at N = 32,
// 9 at N = 16, whatever M), so that one block can take all of K and nothing has to be added up between blocks.
//
// What bounds a step (B200, H = 1024, B = 32): the chain publish -> seen by the other blocks -> shared memory -> tensor core -> gates.
//   * A store by one SM is seen by a relaxed polling load of another after 740 cycles on average, 950 at most; with a release and an
//     acquire on a counter it is 1290 / 1600, and fetching the data behind the counter costs another L2 round trip. So nothing here waits
//     on counters: every word that travels says by itself which step it belongs to. The lowest mantissa bit of a value is one fixed bit that
//     depends on the step and on whether the unit is even: a word of two values ends its halves in (0, 1) or in (1, 0), the other way round at
//     every second use of its place. Words of another step, and words that were cleared, do not have the pattern.
//     The ring has two slots (step parity). Reuse is safe without any further exchange: a block writes step s only after it has
//     read step s - 1 of EVERY block, and each produced that only after it had consumed all of step s - 2. Words of an earlier launch
//     are cleared before the blocks of a direction meet once at the start.
//   * Lines that another SM has just written are slow to read: 128 blocks that read 32 KB each take 1130 cycles when nothing was
//     written, 1406 (the last block 1863) when it was. That is why values travel in 16 bits, and why nothing is polled before it can be
//     there.
//   * Operand A from tensor memory: the instruction then costs what its products cost; from shared memory an M = 128 instruction reads 4 KiB
//     at 128 B per cycle (39 cycles). Weights that do not fit in the 512 columns stay in shared memory (H = 1024: one K tile of 16).
//   * Sixteen warps do everything but issue the MMAs. A warp reads back eight batch columns of the rows of four units, brings them
//     to one (unit, batch) pair per lane through its own 1 KiB of shared memory, and has no other warp to wait for until the words are there. Output
//     stores and prefetches are issued while the words are on their way.
//
// Every wait is bounded by %globaltimer. When a wait runs out the block records a status bit and leaves its loops, and like every block
// waits (bounded) for its own MMAs in flight before it frees its tensor memory and returns.
#include "gru_common.cuh"

#include <algorithm>
#include <atomic>

namespace bc {
namespace gpu {

namespace {

using namespace gru;

constexpr int kWarps = 16;                 // all but the warp that issues the MMAs
constexpr int kWorkers = kWarps * 32;
constexpr int kThreads = kWorkers + 32;
constexpr int kKTile = 64;                 // fp16 elements in one 128-byte swizzle row
constexpr int kMaxParts = 2;                // of the operand, handed to the tensor core one after the other
constexpr int kRows = 128;                 // M
// Read-back through shared memory, [column group][column 8][quarter 4][row 32] words at distances that leave no bank conflicts: a warp writes
// the 32 rows of its quarter, and reads four rows of every quarter in two columns.
constexpr int kBackQuarter = 36, kBackColumn = 4 * kBackQuarter, kBackGroup = 8 * kBackColumn;

// The gate functions are on the critical path of every step and bound by instruction issue: with `tanhf` and IEEE divisions, whose
// rare cases branch, a forward step of H = 1024, B = 32 took 4.34 us, with these 3.69 (with approximate divisions alone 3.68, but tanh
// was then off by up to 4.0 units in the last place for x < 0). Neither may be further off than CUDA's, in no range. Scan of all floats
// against fp64, largest / mean error: tanh up to 0.62 0.84 / 0.25 units (`tanhf` 1.81 / 0.63), 0.62 to 1 1.81 / 0.38 (the same), 1 to 2
// 1.37 / 0.28 (the same); sigmoid as 1 / (1 + __expf(-x)) everywhere: 1.6 for x > 0, 8.4 at -8, 62 at -80, the rounding of x log2 e.
__device__ __forceinline__ float rcp_(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float exp2_(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 1 / (1 + e^-x) as a quarter of the reciprocal of a quarter of the denominator, so that neither leaves the normal range before the
// result does; one step of Newton's method, y + y (1 - d y), takes the approximation's error out.
__device__ __forceinline__ float sigmoidf_(float x) {
  const float d = fmaf(exp2_(x * -1.44269504f), 0.25f, 0.25f);
  const float y = rcp_(d);
  return d < INFINITY ? 0.25f * fmaf(y, fmaf(-d, y, 1.f), y) : y;
}
// sign(x) (1 - 2 / (1 + e^2|x|)); where that cancels, Lambert's continued fraction cut behind its fifth partial denominator as
// x - x v with v = q (315 + 14 q) / (945 + 420 q + 15 q^2), q = x^2: off by 7e-10 at 0.625, and the rounding of v, which is
// below 0.12, hardly shows.
__device__ __forceinline__ float tanhf_(float x) {
  const float q = x * x, a = fabsf(x);
  const bool small = q < 0.39f;
  const float num = small ? q * fmaf(q, 14.f, 315.f) : 2.f;
  const float den = small ? fmaf(q, fmaf(q, 15.f, 420.f), 945.f) : 1.f + exp2_(a * 2.88539008f);
  const float m = small ? a : 1.f;
  return copysignf(fmaf(-m, num * rcp_(den), m), x);
}

// The four warps of a column group have their part of the accumulator in shared memory. It has no limit, so they come to it once per step
// whatever waits have run out.
__device__ __forceinline__ void group_sync(int group) { asm volatile("barrier.cta.sync %0, 128;" ::"r"(group + 1) : "memory"); }

// ---- fp16 operands -------------------------------------------------------------------------------

__device__ __forceinline__ uint16_t half_rn(float v) {
  uint16_t h;
  asm("cvt.rn.f16.f32 %0, %1;" : "=h"(h) : "f"(v));
  return h;
}
__device__ __forceinline__ float half_to_float(uint16_t h) {
  float v;
  asm("cvt.f32.f16 %0, %1;" : "=f"(v) : "h"(h));
  return v;
}
__device__ __forceinline__ float pow2(int e) { return __int_as_float((e + 127) << 23); }
// Bits of a value's place in a word of two: even units in the low half. `phase` alternates between uses of a slot.
__device__ __forceinline__ uint32_t pattern(uint32_t phase) { return phase ? 0x00000001u : 0x00010000u; }
constexpr uint32_t kTagMask = 0x00010001u;
// The fp16 value nearest to h * 2^15 among those that end in `tag`: cut towards zero, and one further from zero if that ends in the other.
__device__ __forceinline__ uint16_t tagged_half(float h, uint32_t tag) {
  uint16_t c;
  asm("cvt.rz.f16.f32 %0, %1;" : "=h"(c) : "f"(h * 32768.f));
  const uint32_t v = h == h ? c : 0x7E00u;             // NaN stays one whatever its last bit
  return (uint16_t)(v + ((v ^ tag) & 1u));
}
__device__ __forceinline__ void st_half(uint16_t* p, uint16_t v) { asm volatile("st.relaxed.gpu.global.u16 [%0], %1;" ::"l"(p), "h"(v) : "memory"); }
__device__ __forceinline__ bool stale(const Words& v, uint32_t pat) {
  uint32_t d = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) d |= v.w[i] ^ pat;
  return (d & kTagMask) != 0;
}
template <int CTAS>
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (CTAS == 1)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
template <int CTAS>
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (CTAS == 1)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// All MMAs issued so far arrive at `bar` of every block that takes part when they are done.
template <int CTAS>
__device__ __forceinline__ void commit(uint32_t bar) {
  if constexpr (CTAS == 1) tc_commit(bar);
  else asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
template <int CTAS>
__device__ __forceinline__ void alloc(uint32_t* slot) {
  if constexpr (CTAS == 1) {
    tmem_alloc(slot, kTmemCols);
  } else {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
}
template <int CTAS>
__device__ __forceinline__ void dealloc(uint32_t tmem) {
  if constexpr (CTAS == 1) tmem_free(tmem, kTmemCols);
  else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}
// All threads of both blocks of a pair.
template <int CTAS>
__device__ __forceinline__ void pair_sync() {
  if constexpr (CTAS == 2) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrival at the barrier at this place in the first block of the pair.
__device__ __forceinline__ void mbar_arrive_first(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .b32 a;\n\t"
      "mapa.shared::cluster.u32 a, %0, 0;\n\t"
      "mbarrier.arrive.shared::cluster.b64 _, [a];\n\t}"
      ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}

// Where everything of one block lives. NB: N of the MMA, at least the batch; CTAS: blocks that share an MMA; H: hidden size.
template <int NB, int CTAS, int H>
struct Plan {
  static constexpr int kTiles = H / kKTile;                                  // K tiles of 64
  // Those whose weights live in tensor memory, behind the accumulator; the others (one, at H = 1024) live in shared memory.
  static constexpr int kTmemTiles = std::min(kTiles, ((int)kTmemCols - NB) / 32);
  static constexpr int kBatchRows = NB / CTAS;                               // batch rows whose words this block brings
  static constexpr int kTileBytes = kBatchRows * 128;
  // A worker's load `it` is the 32-byte word tid + 512 it: sector tid % 4 of batch row tid / 4 % kBatchRows in K tile
  // it * kTilesPerRound + tid / 4 / kBatchRows.
  static constexpr int kTilesPerRound = kWorkers / 4 / kBatchRows;
  static constexpr int kRounds = (kTiles + kTilesPerRound - 1) / kTilesPerRound;
  static constexpr int kParts = std::min(kRounds, kMaxParts);               // what is handed to the tensor core at a time
  static constexpr int kRoundsPerPart = (kRounds + kParts - 1) / kParts;
  static constexpr int kXBytes = kTiles * kTileBytes, kWBytes = (kTiles - kTmemTiles) * kRows * 128;
  // operand, weights, read-back of the warps, scales of the 48 rows, barriers
  static constexpr int kSmem = 1024 + kXBytes + kWBytes + kWarps / 4 * kBackGroup * 4 + 256 + 128;
};

// Sixteen weights of a row times its scale as pairs of fp16: the upper part, or what it leaves.
__device__ __forceinline__ void split16(const float* p, float scale, bool lower, uint32_t* o) {
  uint16_t h[16];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float4 f = __ldg(reinterpret_cast<const float4*>(p) + i);
    const float v[4] = {f.x * scale, f.y * scale, f.z * scale, f.w * scale};
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const uint16_t hi = half_rn(v[e]);
      // an infinite weight has no lower part
      h[4 * i + e] = !lower ? hi : (hi & 0x7C00u) == 0x7C00u ? (uint16_t)0 : half_rn(v[e] - half_to_float(hi));
    }
  }
#pragma unroll
  for (int i = 0; i < 8; i++) o[i] = h[2 * i] | (uint32_t)h[2 * i + 1] << 16;
}

// NB: N of the MMA (16 or 32, at least the batch). CTAS = 2: the two blocks of a cluster share an MMA of M = 256. Each brings the words of half of the batch
// into its shared memory, and the tensor cores of both read both halves.
template <int NB, int CTAS, int H>
__global__ void __launch_bounds__(kThreads, 1) gru_forward_kernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);       // the same for all lanes, and known to be
  const int dir = blockIdx.y, u0 = blockIdx.x * kUnits;
  const int T = p.d.T, B = p.d.B, ND = p.d.ndir;
  using pl = Plan<NB, CTAS, H>;
  const int rank = CTAS == 1 ? 0 : blockIdx.x & 1;

  uint8_t* x_s = smem;
  uint8_t* w_s = x_s + pl::kXBytes;
  float* back_s = reinterpret_cast<float*>(w_s + pl::kWBytes);          // read-back
  float* scale_s = back_s + kWarps / 4 * kBackGroup;                              // [gate][unit]: power of two of each row
  uint64_t* bar_s = reinterpret_cast<uint64_t*>(scale_s + 64);         // full[kMaxParts], done, drain
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_s + kMaxParts + 2);
  volatile int* abort_s = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t full_bar = smem_u32(bar_s), done_bar = full_bar + 8 * kMaxParts, drain_bar = done_bar + 8;
  const uint32_t x_addr = smem_u32(x_s), w_addr = smem_u32(w_s);

  if (tid == 0) {
    for (int i = 0; i < kMaxParts; i++) mbar_init(full_bar + 8 * i, kWarps + (rank == 0 ? CTAS - 1 : 0));
    mbar_init(done_bar, 1);
    mbar_init(drain_bar, 1);
    *abort_s = 0;
    mbar_init_fence();
  }
  if (warp == kWarps) alloc<CTAS>(tmem_slot);

  // The part of the ring that this block writes, cleared in both slots. The ring of a direction and slot is [K tile][batch NB][64].
  const uint32_t slot_halves = (uint32_t)pl::kTiles * NB * kKTile;
  uint16_t* ring = reinterpret_cast<uint16_t*>(p.ring) + (size_t)dir * 2 * slot_halves;
  uint16_t* mine = ring + (size_t)(u0 / kKTile) * NB * kKTile + u0 % kKTile;
  for (int i = tid; i < 2 * B * kUnits; i += kThreads)
    st_half(mine + (i & 1 ? slot_halves : 0u) + (i / 2 / kUnits) * kKTile + i / 2 % kUnits, 0);
  for (int i = tid; i < pl::kXBytes / 16; i += kThreads) reinterpret_cast<uint4*>(x_s)[i] = make_uint4(0, 0, 0, 0);

  // Scale of every row. Infinite weights and NaN are left out of the maximum: they stay what they are.
  const float* w = p.w_hh[dir];
  if (warp < kWarps)
    for (int r = warp; r < 3 * kUnits; r += kWarps) {
      const float4* row = reinterpret_cast<const float4*>(w + (size_t)(r / kUnits * H + u0 + r % kUnits) * H);
      uint32_t m = 0;
      for (int i = lane; i < H / 4; i += 32) {
        const float4 v = __ldg(row + i);
        const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const uint32_t b = __float_as_uint(f[e]) & 0x7FFFFFFFu;
          if (b < 0x7F800000u) m = max(m, b);
        }
      }
      m = __reduce_max_sync(0xffffffffu, m);
      const int e = m ? max((int)(m >> 23) - 127, -90) : 14;
      if (lane == 0) scale_s[r] = pow2(14 - e);
    }
  fence_proxy_async();
  __threadfence();
  tc_fence_before();
  __syncthreads();
  pair_sync<CTAS>();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  Meeting meeting{};
  if (tid == 0) meeting = meet_arrive(p, dir, gridDim.x);

  // Row (lane of tensor memory) 32 q + 16 part + 4 gate + i holds unit 4 q + i: part 0 the upper, part 1 the lower halves.
  const int quarter = warp & 3, part = lane >> 4, gate = (lane & 15) >> 2;
  if (warp < kWarps) {
    const bool row_ok = gate < 3;
    const int unit = 4 * quarter + (lane & 3);
    const float* row = w + (size_t)((row_ok ? gate : 0) * H + u0 + unit) * H;
    const float scale = row_ok ? scale_s[gate * kUnits + unit] : 0.f;
    for (int kt = warp >> 2; kt < pl::kTiles; kt += kWarps / 4) {
      uint32_t v[32];
#pragma unroll
      for (int c = 0; c < 4; c++) {
        if (row_ok) split16(row + kt * kKTile + 16 * c, scale, part != 0, v + 8 * c);
        else
#pragma unroll
          for (int i = 0; i < 8; i++) v[8 * c + i] = 0;
      }
      __syncwarp();
      if (kt < pl::kTmemTiles) {
        const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(NB + kt * 32);
        tmem_st16(at, reinterpret_cast<const float*>(v));
        tmem_st16(at + 16, reinterpret_cast<const float*>(v + 16));
      } else {
        const int r = quarter * 32 + lane;
        uint8_t* o = w_s + ((kt - pl::kTmemTiles) * kRows + r) * 128;
#pragma unroll
        for (int c = 0; c < 8; c++) reinterpret_cast<uint4*>(o)[c ^ (r & 7)] = make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
      }
    }
    tmem_st_wait();
    fence_proxy_async();
  }
  bool ok = true;
  if (tid == 0) ok = meet_wait(p, meeting);
  tc_fence_before();
  ok = __syncthreads_and(ok) != 0;
  tc_fence_after();

  auto give_up = [&](uint32_t why) {
    atomicOr(p.status, why);
    *abort_s = 1;
    return false;
  };
  if (ok && warp == kWarps) {
    // ---------------- the warp that issues the MMAs ----------------
    const bool leader = elect_one();
    const uint32_t idesc = (1u << 4) | ((uint32_t)(NB >> 3) << 17) | ((uint32_t)(CTAS * kRows >> 4) << 24);     // fp16 operands, fp32 accumulator
    const uint64_t b_desc = operand_desc(x_addr), a_desc = operand_desc(w_addr);
    for (int s = 1; ok && s < T; s++) {
#pragma unroll
      for (int g = 0; g < pl::kParts; g++) {
        ok = ok && bar_wait(full_bar + 8 * g, (uint32_t)(s - 1) & 1, 4 * p.timeout_ns, abort_s);
        if (!ok) break;
        if (CTAS == 2 && rank != 0) {            // this block's half is there
          if (elect_one()) mbar_arrive_first(full_bar + 8 * g);
          __syncwarp();
          continue;
        }
        if (g == 0) tc_fence_after();
        // Straight-line code: with a branch among them an instruction takes 30 cycles to issue instead of 12.
        if (elect_one()) {
          constexpr int kTilesPerPart = pl::kRoundsPerPart * pl::kTilesPerRound;
#pragma unroll
          for (int kt = g * kTilesPerPart; kt < (g + 1) * kTilesPerPart; kt++) {
            if (kt >= pl::kTiles) break;
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
              const uint64_t b = b_desc + (uint64_t)(kt * pl::kTileBytes / 16 + 2 * ks);
              if (kt < pl::kTmemTiles) mma_ts<CTAS>(tmem, tmem + NB + kt * 32 + 8 * ks, b, idesc, kt + ks > 0);
              else mma_ss<CTAS>(tmem, a_desc + (uint64_t)((kt - pl::kTmemTiles) * kRows * 8 + 2 * ks), b, idesc, 1);
            }
          }
        }
        __syncwarp();
      }
      if (rank == 0 && elect_one()) commit<CTAS>(done_bar);
      __syncwarp();
    }
    if (leader) {
      if (!ok && !*abort_s) give_up(kGruTimeoutBlock);
      // Nothing may be in flight when tensor memory is freed, whatever this or another warp has not waited for.
      if (rank == 0) {
        commit<CTAS>(drain_bar);
        mbar_drain(drain_bar, 0);
      }
    }
    __syncwarp();
  } else if (ok) {
    // ---------------- workers ----------------
    const int sector = tid & 3, row = tid >> 2, xrow = row % pl::kBatchRows, xb = rank * pl::kBatchRows + xrow, kt0 = row / pl::kBatchRows;
    const uint32_t dst = x_addr + (uint32_t)(row * 128 + (((2 * sector) ^ (xrow & 7)) << 4));
    const uint32_t* src0 = reinterpret_cast<const uint32_t*>(ring) + (size_t)(kt0 * NB + xb) * (kKTile / 2) + sector * 8;
    constexpr uint32_t kRoundBytes = kWorkers * 32, kRoundWords = pl::kTilesPerRound * NB * kKTile / 2;   // in shared memory, in the ring
    const int loads = xb < B && kt0 < pl::kTiles ? (pl::kTiles - kt0 + pl::kTilesPerRound - 1) / pl::kTilesPerRound : 0;

    // Gates: unit u of the block, batch entry b. The four warps of a column group read eight columns back, each those of its quarter of the
    // rows, and share them through shared memory. The next step writes those only when all warps have brought their words of it.
    const int u = lane & 15, b = 2 * warp + (lane >> 4), group = warp >> 2;
    const bool gates = 8 * group < B;                     // of the column group
    const bool active = b < B;
    float* back_w = back_s + group * kBackGroup + quarter * kBackQuarter + lane;
    const float* back_r = back_s + group * kBackGroup + (b & 7) * kBackColumn + (u >> 2) * kBackQuarter + (u & 3);
    float inv[3], bias[3];
#pragma unroll
    for (int g = 0; g < 3; g++) {
      // 1 / (scale of the row * 2^15): scales are powers of two
      inv[g] = __int_as_float(((254 - 15) << 23) - __float_as_int(scale_s[g * kUnits + u]));
      bias[g] = p.b_hh[dir][g * H + u0 + u];
    }
    const ptrdiff_t step = dir ? -1 : 1;
    const int t_first = dir ? T - 1 : 0, bb = active ? b : 0;
    const int gx_row = ND * 3 * H, y_row = ND * H;
    const float* gx_p = p.gx + ((size_t)t_first * B + bb) * gx_row + dir * 3 * H + u0 + u;
    float* y_p = p.y + ((size_t)t_first * B + bb) * y_row + dir * H + u0 + u;
    float4* rsv_p = p.rsv ? p.rsv + ((size_t)(dir * T + t_first) * B + bb) * H + u0 + u : nullptr;
    float* fac_p = p.fac ? p.fac + ((size_t)(dir * T + t_first) * B + bb) * 5 * H + u0 + u : nullptr;
    uint16_t* out = mine + bb * kKTile + u;
    const bool stamping = p.prof && tid == 0 && blockIdx.x == 0 && blockIdx.y == 0;
    auto stamp = [&](int s, int i) {
      if (stamping) p.prof[(size_t)s * 8 + i] = gtimer();
    };
    float gx[3] = {0.f, 0.f, 0.f}, h = 0.f;
    auto load_gx = [&]() {
      if (active) {
#pragma unroll
        for (int g = 0; g < 3; g++) gx[g] = __ldg(gx_p + g * H);
      }
      gx_p += step * B * gx_row;
    };
    load_gx();
    // Cycles from this block's publication to its first poll. A poll that finds nothing costs as much as one that brings the operand, for all
    // blocks; a late one delays its own. us per step without / with 300 / with this rule: H = 1024, B = 32 3.13 / 2.85 / 2.73, B = 8 2.18 /
    // 1.99 / 1.97, H = 512, B = 3 1.50 / 1.55 / 1.50, H = 128, B = 8 1.27 / 1.39 / 1.28. Warps without gates come here 300 cycles earlier.
    const uint32_t volume = (uint32_t)(min(B, pl::kBatchRows) * H * 2);
    const uint32_t pause = (CTAS == 2 ? 600 : min(volume / 40, 400u)) + (gates ? 0 : 300);
    bool good = true;
    for (int s = 0; s < T; s++) {
      stamp(s, 0);
      float acc[3] = {0.f, 0.f, 0.f};
      if (s > 0) {
        if (good && !bar_wait(done_bar, (uint32_t)(s - 1) & 1, 4 * p.timeout_ns, abort_s)) good = *abort_s ? false : give_up(kGruTimeoutMma);
        good = __all_sync(0xffffffffu, good) != 0;
        stamp(s, 1);
        if (gates) {
          uint32_t v[8];
          tc_fence_after();
          tmem_ld8(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(8 * (warp >> 2)), v);
          tc_fence_before();
#pragma unroll
          for (int c = 0; c < 8; c++) back_w[c * kBackColumn] = __uint_as_float(v[c]);
          group_sync(group);
#pragma unroll
          for (int g = 0; g < 3; g++) acc[g] = back_r[g * 4] + back_r[16 + g * 4];
        }
      }
      stamp(s, 2);
      const uint32_t phase = (uint32_t)(s >> 1) & 1;       // of the words that this step publishes
      if (gates) {
        const float hn = fmaf(acc[2], inv[2], bias[2]);
        const float r_ = sigmoidf_(fmaf(acc[0], inv[0], gx[0] + bias[0]));
        const float z = sigmoidf_(fmaf(acc[1], inv[1], gx[1] + bias[1]));
        const float n = tanhf_(gx[2] + r_ * hn);
        const float hp = h;
        h = n + z * (h - n);
        if (active) {
          if (s + 1 < T) st_half(out + ((s & 1) ? slot_halves : 0u), tagged_half(h, phase ^ (uint32_t)(u & 1)));
          stamp(s, 3);
          // The other blocks do not wait for what follows.
          *y_p = h;
          if (rsv_p) *rsv_p = make_float4(r_, z, n, hn);
          if (fac_p) {
            const Factors f = factors(make_float4(r_, z, n, hn), hp);
            fac_p[0] = f.r; fac_p[H] = f.z; fac_p[2 * H] = f.nr; fac_p[3 * H] = f.n; fac_p[4 * H] = f.keep;
          }
        }
        y_p += step * B * y_row;
        if (rsv_p) rsv_p += step * B * H;
        if (fac_p) fac_p += step * B * 5 * H;
        if (s + 1 < T) load_gx();
      }
      if (s + 1 == T) break;
      stamp(s, 4);
      for (const uint32_t c0 = clock32(); clock32() - c0 < pause;) {
      }
      stamp(s, 5);
      // The operand of the next step. All of a thread's loads are in flight together; a warp hands over the rounds as they are complete.
      const uint32_t pat = pattern(phase);
      const uint32_t* src = src0 + ((s & 1) ? slot_halves / 2 : 0u);
      Words v[pl::kRounds];
#pragma unroll
      for (int i = 0; i < pl::kRounds; i++)
        if (i < loads) ld_words(src + i * kRoundWords, v[i]);
      uint32_t spins = 0, left = good ? (1u << pl::kRounds) - 1 : 0;
      unsigned long long t0 = 0;
      while (left) {
#pragma unroll
        for (int i = 0; i < pl::kRounds; i++) {
          if (left >> i & 1) {
            const bool missing = i < loads && stale(v[i], pat);
            if (__any_sync(0xffffffffu, missing)) {
              if (missing) ld_words(src + i * kRoundWords, v[i]);
            } else {
              if (i < loads) st_shared2(dst + i * kRoundBytes, v[i]);
              fence_proxy_async();
              __syncwarp();
              left &= ~(1u << i);
              constexpr uint32_t kOfPart = (1u << pl::kRoundsPerPart) - 1;
              if ((left >> (i / pl::kRoundsPerPart * pl::kRoundsPerPart) & kOfPart) == 0 && lane == 0) mbar_arrive(full_bar + 8 * (i / pl::kRoundsPerPart));
            }
          }
        }
        if (((++spins) & 63) == 0) {
          const unsigned long long now = gtimer();
          if (t0 == 0) t0 = now;
          if (*abort_s) good = false;
          else if (now - t0 > p.timeout_ns) good = give_up(kGruTimeoutGrid);
          if (!__all_sync(0xffffffffu, good)) {
            good = false;
            break;
          }
        }
      }
      stamp(s, 6);
    }
  }

  tc_fence_before();
  __syncthreads();
  pair_sync<CTAS>();                       // neither block leaves while the other may still read its memory or arrive at its barriers
  if (warp == kWarps) dealloc<CTAS>(tmem);
}

template <int NB, int CTAS, int H>
cudaError_t launch_with(const Params& p, cudaStream_t stream) {
  auto kernel = gru_forward_kernel<NB, CTAS, H>;
  const int smem = std::max(Plan<NB, CTAS, H>::kSmem, kMinSmem);
  // The attribute belongs to a device: set once for each, to all that a block can have.
  static std::atomic<uint64_t> granted{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 64 || !(granted.load(std::memory_order_relaxed) >> dev & 1)) {
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024)) != cudaSuccess) return e;
    if (dev < 64) granted.fetch_or(1ull << dev, std::memory_order_relaxed);
  }
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = CTAS;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(H / kUnits, p.d.ndir);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = CTAS > 1 ? 2 : 1;
  if (CTAS > 1) {                             // asked beforehand: a launch that fails would end a capture
    int n = 0;
    cfg.numAttrs = 2;
    if ((e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg)) != cudaSuccess) return e;
    if (n * CTAS < H / kUnits * p.d.ndir) return cudaErrorCooperativeLaunchTooLarge;
  }
  return cudaLaunchKernelEx(&cfg, kernel, p);
}

template <int NB, int CTAS>
cudaError_t launch(const Params& p, cudaStream_t stream) {
  switch (p.d.H) {
    case 128: return launch_with<NB, CTAS, 128>(p, stream);
    case 256: return launch_with<NB, CTAS, 256>(p, stream);
    case 384: return launch_with<NB, CTAS, 384>(p, stream);
    case 512: return launch_with<NB, CTAS, 512>(p, stream);
    case 640: return launch_with<NB, CTAS, 640>(p, stream);
    case 768: return launch_with<NB, CTAS, 768>(p, stream);
    case 896: return launch_with<NB, CTAS, 896>(p, stream);
    case 1024: return launch_with<NB, CTAS, 1024>(p, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

namespace gru {

// Pairs halve what a block has to read and pay for it with a meeting of the two in every step. us per step at B = 32, single / pairs: H = 1024
// 3.21 / 2.73, 768 2.69 / 2.44, 512 2.40 / 2.37, 256 1.85 / 1.94, 128 1.62 / 1.65. Up to 16 batch entries an MMA of N = 16 costs
// 9 cycles instead of 16, and a pair has none of N = 16.
cudaError_t launch_forward(const Params& p, cudaStream_t stream) {
  if (p.d.B <= 16) return launch<16, 1>(p, stream);
  if (p.d.H >= 512) {
    const cudaError_t e = launch<32, 2>(p, stream);
    if (e != cudaErrorCooperativeLaunchTooLarge) return e;      // pairs that do not fit beside each other
  }
  return launch<32, 1>(p, stream);
}

}  // namespace gru
}  // namespace gpu
}  // namespace bc

// Persistent bidirectional GRU layer for sm_100a (see gru_persistent.h for the interface).
//
// Work split. Direction d of a layer is run by H/16 blocks (grid.y = direction); block c owns
// the hidden units [16c, 16c+16) and produces their outputs. For the recurrent product the blocks
// work in groups of C that split the reduction length K among themselves: block q of a group keeps,
// for ALL units of its group, the weight columns of its K range on chip for the whole sequence
// (forward 48C rows x H/C columns, backward 16C rows x 3H/C columns: 192 KiB of fp32 at H = 1024
// either way). Each time step it
//   1. polls its K range of the operand of this step (h_{t-1} forward, the pre-activation gradients
//      backward) in a ring in global memory, and puts it into shared memory in the 128-byte swizzle,
//   2. multiplies with tcgen05.mma (TF32 operands): the weights are the M side and live in TENSOR
//      MEMORY, the batch is the N side, K = 8 per instruction, accumulator in tensor memory,
//   3. reads the accumulator back (tcgen05.ld: a lane is a weight row, a column a batch entry) and
//      sends every other member of the group the partial sums of that member's units,
//   4. adds up the C partial sums of its own units, applies the gate non-linearities (forward) or
//      forms the next pre-activation gradients (backward), and puts them into the ring.
//
// What bounds a step, and what was done about it (B200, H = 1024, B = 32, cycles at 1.9 GHz):
//   * A store by one SM is seen by a relaxed polling load of another after 740 cycles on average, 950
//     at most; with a release and an acquire on a counter it is 1290 / 1600, and fetching the data
//     behind the counter costs another L2 round trip. So nothing here waits on counters: every word
//     that travels says by itself which step it belongs to.
//       - Operand words. tcgen05 reads 19 bits of a TF32 operand and ignores the low 13 bits of
//         its 32-bit container; those carry the step number. The reader compares them and stores
//         the word as it is. (The full fp32 value goes to the output tensor as well.)
//       - Partial sums need all 32 bits: three of them and the step number share a 16-byte word
//         that is written and read as one access (.b128, single-copy atomic).
//     Both areas have two slots (step parity). Slot reuse is safe without any further exchange: a
//     block writes step s only after partial sums or operand words of step s - 1 from its group, which
//     together depend on step s - 1 of EVERY block, and a block produces step s - 1 only after it
//     has consumed all of step s - 2. Stale words of an earlier launch are cleared before the blocks
//     of a direction meet once at the start.
//   * Operand A from tensor memory: one M = 128, N = 32, K = 8 instruction takes 20 cycles, from shared
//     memory 45 (it reads 5 KiB at 128 B per cycle). Weights that do not fit in the 512 columns
//     (forward groups of four at H = 1024) stay in shared memory.
//   * The MMAs are issued by an elected lane of a warp of its own; issued from under a
//     `threadIdx.x == n` branch the same M = 64, N = 32 instruction took 55 cycles instead of 26.
// One layer (T = 350, B = 32, H = 1024, both directions): see the figures at choose_split().
//
// Every wait is bounded by %globaltimer. When a wait runs out the block records a status bit, waits
// (bounded) for its own MMAs in flight, frees its tensor memory and returns.
#include "gru_persistent.h"

#include <stdlib.h>

#include <algorithm>
#include <atomic>

namespace bc {
namespace gpu {

namespace {

constexpr int kUnits = 16;            // hidden units per block
constexpr int kKTile = 32;            // fp32 elements in one 128-byte swizzle row
constexpr int kWorkers = 256;         // eight warps: operand loads, accumulator read-back, exchange, gate math
constexpr int kThreads = kWorkers + 32;   // plus the warp that issues the MMAs
constexpr int kMaxBlocksPerDir = 64;  // H / 16 at H = 1024
constexpr int kTmemCols = 512;
constexpr int kLoadsPerGroup = 4;     // operand loads of a thread per pipeline group (one mbarrier each)
constexpr int kMaxGroups = 7;         // of a step: 28 K tiles of 32 batch rows, H = 896 unsplit
constexpr int kMinSmem = 120 * 1024;  // more than half of an SM's shared memory: one block per SM, since a block takes all of tensor memory

struct Params {
  GruDims d;
  const float* w_hh[2];   // [3H, H] of each direction
  const float* b_hh[2];   // forward: [3H] of each direction
  const float* gx;        // forward
  float* y;               // forward: out; backward: in (const)
  float4* rsv;            // forward: out, or null; backward: in
  const float* dy;        // backward
  float* dg;              // backward: out
  float* db;              // backward: out
  uint32_t* ring;         // operand words: [dir][slot 2][member C][K tile][batch B][32]
  uint4* xchg;            // partial sums: [dir][owner block][source C][slot 2][pack][row] x 16 bytes
  uint32_t* sync;         // per direction: arrivals, generation
  uint32_t* status;
  unsigned long long timeout_ns;
  unsigned long long* prof;   // optional: 8 time stamps per step of block (0, 0), for tuning
};

// ---- PTX wrappers ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded wait for the phase with the given parity; also gives up when `abort_flag` is raised.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, unsigned long long timeout_ns, const volatile int* abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = gtimer();
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if (((++spins) & 63) == 0) {
      if (abort_flag && *abort_flag) return false;
      if (gtimer() - t0 > timeout_ns) return false;
    }
  }
  return true;
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// D[m, n] (+)= A[m, k] * B[n, k], A in tensor memory / in shared memory.
__device__ __forceinline__ void tc_mma_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_mma_ss(uint32_t d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// N consecutive columns of this thread's tensor-memory lane.
template <int N> __device__ __forceinline__ void tc_ld(uint32_t taddr, uint32_t* r);
template <> __device__ __forceinline__ void tc_ld<16>(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
template <> __device__ __forceinline__ void tc_ld<32>(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const float* v) {
  const uint32_t* r = reinterpret_cast<const uint32_t*>(v);
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}

// Words that travel between blocks.
__device__ __forceinline__ void st_word(uint32_t* p, uint32_t v) { asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ uint4 ld_words(const uint32_t* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_pack(uint4* p, uint4 v) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\t.reg .b64 lo, hi;\n\t"
      "mov.b64 lo, {%1, %2};\n\tmov.b64 hi, {%3, %4};\n\tmov.b128 t, {lo, hi};\n\t"
      "st.relaxed.gpu.global.b128 [%0], t;\n\t}"
      ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint4 ld_pack(const uint4* p) {
  uint4 v;
  asm volatile(
      "{\n\t.reg .b128 t;\n\t.reg .b64 lo, hi;\n\t"
      "ld.relaxed.gpu.global.b128 t, [%4];\n\t"
      "mov.b128 {lo, hi}, t;\n\tmov.b64 {%0, %1}, lo;\n\tmov.b64 {%2, %3}, hi;\n\t}"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
constexpr uint32_t kTagMask = 0x1FFFu;
__device__ __forceinline__ uint32_t tagged(float v, uint32_t tag) { return (__float_as_uint(v) & ~kTagMask) | tag; }
__device__ __forceinline__ bool stale(const uint4& v, uint32_t tag) {
  return (((v.x ^ tag) | (v.y ^ tag) | (v.z ^ tag) | (v.w ^ tag)) & kTagMask) != 0;
}

// Shared-memory matrix descriptor of a K-major operand tile stored as rows of 128 bytes with the
// 128-byte swizzle (16-byte chunk c of row r sits at chunk c ^ (r & 7)): groups of 8 rows are 1024
// bytes apart; the leading-dimension offset is unused because a tile is one swizzle atom wide.
__device__ __forceinline__ uint64_t operand_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);   // start address
  d |= (uint64_t)(1024u >> 4) << 32;              // stride between 8-row groups
  d |= (uint64_t)1 << 46;                         // descriptor version of sm_100
  d |= (uint64_t)2 << 61;                         // 128-byte swizzle
  return d;
}

__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + __expf(-x)); }

// Barrier of the eight worker warps that also tells whether all of them are still fine.
__device__ __forceinline__ bool workers_sync_and(bool ok) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, 1, 256, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r) : "r"((uint32_t)ok) : "memory");
  return r != 0;
}

// Where everything of one block lives; a function of the pass, the split and the dimensions.
struct Plan {
  int kq;            // K range of a member: columns of the recurrent weights it holds
  int ntile;         // K tiles of 32 (the last one may be half)
  int m0, m1;        // M of the accumulator tiles (m1 = 0: one tile); rows beyond the group's are padding
  int col0;          // first tensor-memory column of the weights; the accumulators lie below
  int kt0, kt1;      // K columns of either tile that live in tensor memory; the others live in shared memory
  int x_bytes, w_bytes, own_bytes;
  __host__ __device__ int smem() const { return 1024 + x_bytes + w_bytes + own_bytes + 256; }
};
template <bool BWD> struct RowsPerOwner { static constexpr int value = BWD ? kUnits : 3 * kUnits; };

template <bool BWD>
__host__ __device__ inline Plan make_plan(int C, int nb, int H) {
  Plan p;
  const int rows = RowsPerOwner<BWD>::value * C;
  p.kq = (BWD ? 3 * H : H) / C;
  p.ntile = (p.kq + kKTile - 1) / kKTile;
  p.m0 = rows > 64 ? 128 : 64;
  p.m1 = rows > 128 ? (rows > 192 ? 128 : 64) : 0;
  p.col0 = p.m1 ? 2 * nb : nb;
  int room = kTmemCols - p.col0;
  p.kt0 = p.kq <= room ? p.kq : room / kKTile * kKTile;
  room -= p.kt0;
  p.kt1 = !p.m1 ? 0 : p.kq <= room ? p.kq : room / kKTile * kKTile;
  p.x_bytes = p.ntile * nb * 128;
  p.w_bytes = ((p.kq - p.kt0 + kKTile - 1) / kKTile * p.m0 + (p.m1 ? (p.kq - p.kt1 + kKTile - 1) / kKTile * p.m1 : 0)) * 128;
  p.own_bytes = RowsPerOwner<BWD>::value * (nb + 1) * 4;
  return p;
}
__host__ __device__ inline int packs_of(int batch) { return (batch + 2) / 3; }   // three partial sums and the step number per 16 bytes

// The 16 weights of row `r` of the group at columns k0 .. k0 + 15 of member q's K range (k0 a multiple of 16).
//   forward : rows ordered owner, gate, unit; K = hidden units            W[g * H + unit][q * kq + k]
//   backward: rows ordered owner, unit; K ordered gate, unit of the range   W[g * H + unit'][unit]
// A run of 16 columns stays inside one gate, because a member's range of units is a multiple of 16.
template <bool BWD>
__device__ __forceinline__ void load_weights16(const float* w, int H, int C, int grp, int q, int kq, int r, int k0, float* o) {
  if (!BWD) {
    const int m = r / 48, g = (r % 48) / kUnits, u = r % kUnits;
    const float4* p = reinterpret_cast<const float4*>(w + (size_t)(g * H + (grp * C + m) * kUnits + u) * H + q * kq + k0);
#pragma unroll
    for (int i = 0; i < 4; i++) reinterpret_cast<float4*>(o)[i] = __ldg(p + i);
  } else {
    const int range = H / C, g = k0 / range, kk = q * range + k0 - g * range;
    const float* p = w + (size_t)(g * H + kk) * H + grp * C * kUnits + r;
#pragma unroll
    for (int i = 0; i < 16; i++) o[i] = __ldg(p + (size_t)i * H);
  }
}

// Inputs of one backward step for the (unit, batch) pairs of a thread.
struct BwdInputs {
  float4 a[3];          // r, z, n, W_hn h + b_hn
  float hp[3], dy[3];
};

__device__ __forceinline__ void load_bwd_inputs(const Params& p, BwdInputs& in, int t, int dir, int unit, int b0, int nb) {
  const int T = p.d.T, B = p.d.B, H = p.d.H, ND = p.d.ndir;
  const int tprev = dir ? t + 1 : t - 1;
  const bool has_prev = tprev >= 0 && tprev < T;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    if (j < nb) {
      const int b = b0 + j;
      in.a[j] = __ldg(p.rsv + ((size_t)(dir * T + t) * B + b) * H + unit);
      in.hp[j] = has_prev ? __ldg(p.y + ((size_t)tprev * B + b) * (ND * H) + dir * H + unit) : 0.f;
      in.dy[j] = __ldg(p.dy + ((size_t)t * B + b) * (ND * H) + dir * H + unit);
    }
  }
}

// BWD: pass; C: blocks per group; NB: N of the MMA (16 or 32, at least the batch).
template <bool BWD, int C, int NB>
__global__ void __launch_bounds__(kThreads, 1) gru_persistent_kernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);

  constexpr int kRows = RowsPerOwner<BWD>::value;
  constexpr int R = kRows * C;
  constexpr int kGates = BWD ? 1 : 3;      // accumulator rows per unit
  constexpr int kOwnStride = NB + 1;
  constexpr int kGateWords = BWD ? 3 : 1;  // operand words that a (unit, batch) pair publishes per step
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int dir = blockIdx.y, u0 = blockIdx.x * kUnits;
  const int T = p.d.T, B = p.d.B, H = p.d.H, ND = p.d.ndir;
  const int nblocks = gridDim.x;
  const int grp = blockIdx.x / C, q = blockIdx.x % C;
  const Plan pl = make_plan<BWD>(C, NB, H);
  const int npacks = packs_of(B);

  uint8_t* x_s = smem;
  uint8_t* w_s = smem + pl.x_bytes;
  float* own_s = reinterpret_cast<float*>(w_s + pl.w_bytes);                       // this block's own rows of the accumulator
  uint64_t* bar_s = reinterpret_cast<uint64_t*>(w_s + pl.w_bytes + pl.own_bytes);  // full[kMaxGroups], done, drain
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_s + kMaxGroups + 2);
  volatile int* abort_s = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t full_bar = smem_u32(bar_s), done_bar = full_bar + 8 * kMaxGroups, drain_bar = done_bar + 8;
  const uint32_t x_addr = smem_u32(x_s), w_addr = smem_u32(w_s);

  if (tid == 0) {
    for (int i = 0; i < kMaxGroups; i++) mbar_init(full_bar + 8 * i, kWorkers / 32);
    mbar_init(done_bar, 1);
    mbar_init(drain_bar, 1);
    *abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kWorkers / 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }

  // The part of the ring that this block writes (both slots) and the partial sums that it will
  // receive: cleared, so that nothing of an earlier launch passes for a word of this one.
  const int range = H / C;                                       // units of one member's K range
  const uint32_t ring_member = (uint32_t)pl.ntile * B * kKTile;  // words of one member's range and slot
  const uint32_t ring_slot = ring_member * C;
  uint32_t* ring = p.ring + (size_t)dir * 2 * ring_slot;
  // word of (gate g, unit u0 + u, batch b): member u0 / range, column g * range + u0 % range + u
  const uint32_t my_member = (uint32_t)(u0 / range) * ring_member;
  const int my_col = u0 % range;
  auto ring_at = [&](int g, int u, int b) -> uint32_t {
    const int k = g * range + my_col + u;
    return my_member + (uint32_t)((k >> 5) * B + b) * kKTile + (k & 31);
  };
  const int xslot = npacks * kRows;                              // 16-byte words of one tile and slot
  uint4* xin = p.xchg + ((size_t)dir * nblocks + blockIdx.x) * C * 2 * xslot;
  for (int i = tid; i < kGateWords * kUnits * B; i += kThreads) {
    const int u = i % kUnits, b = i / kUnits % B, g = i / (kUnits * B);
    st_word(ring + ring_at(g, u, b), 0u);
    st_word(ring + ring_slot + ring_at(g, u, b), 0u);
  }
  if (C > 1)
    for (int i = tid; i < C * 2 * xslot; i += kThreads) st_pack(xin + i, make_uint4(0, 0, 0, 0));
  for (int i = tid; i < pl.x_bytes / 16; i += kThreads) reinterpret_cast<uint4*>(x_s)[i] = make_uint4(0, 0, 0, 0);
  fence_proxy_async();
  __threadfence();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  uint32_t* cnt = p.sync + dir * 32;
  volatile uint32_t* gen = p.sync + dir * 32 + 16;
  uint32_t my_gen = 0;
  if (tid == 0) {
    my_gen = *gen;               // read before this block's arrival: cannot move on until it has arrived
    __threadfence();
    if (atomicAdd(cnt, 1u) == (uint32_t)nblocks - 1) {
      *(volatile uint32_t*)cnt = 0;
      __threadfence();
      *gen = my_gen + 1;
    }
  }

  // The group's weight rows for this block's K range, resident for the whole sequence. In a tile with
  // M = 128 row r is lane r of tensor memory; with M = 64 it is lane (r / 16) * 32 + r % 16.
  const float* w = p.w_hh[dir];
  if (warp < kWorkers / 32) {
    const int quarter = warp & 3;
    for (int tile = 0; tile < (pl.m1 ? 2 : 1); tile++) {
      const int m = tile ? pl.m1 : pl.m0, kt = tile ? pl.kt1 : pl.kt0;
      const int r = tile * 128 + (m == 128 ? quarter * 32 + lane : quarter * 16 + (lane & 15));
      const bool valid = r < R && (m == 128 || lane < 16);
      for (int k0 = 16 * (warp >> 2); k0 < kt; k0 += 32) {
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = 0.f;
        if (valid) load_weights16<BWD>(w, H, C, grp, q, pl.kq, r, k0, v);
        __syncwarp();
        tc_st16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(pl.col0 + (tile ? pl.kt0 : 0) + k0), v);
      }
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    uint8_t* dst = w_s;
    for (int tile = 0; tile < (pl.m1 ? 2 : 1); tile++) {
      const int m = tile ? pl.m1 : pl.m0, kt = tile ? pl.kt1 : pl.kt0;
      const int runs = (pl.kq - kt) / 16;
      for (int i = tid; i < m * runs; i += kWorkers) {
        const int rt = i % m, r = tile * 128 + rt, k = (i / m) * 16;      // counted from kt
        float v[16];
#pragma unroll
        for (int e = 0; e < 16; e++) v[e] = 0.f;
        if (r < R) load_weights16<BWD>(w, H, C, grp, q, pl.kq, r, kt + k, v);
        uint8_t* row = dst + ((k >> 5) * m + rt) * 128;
#pragma unroll
        for (int e = 0; e < 4; e++)
          reinterpret_cast<float4*>(row)[(((k & 31) >> 2) + e) ^ (rt & 7)] = make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
      }
      dst += (runs + 1) / 2 * m * 128;
    }
    fence_proxy_async();
  }
  bool ok = true;
  if (tid == 0) {
    const unsigned long long t0 = gtimer();
    uint32_t spins = 0;
    while (*gen == my_gen) {
      if (((++spins) & 31) == 0 && gtimer() - t0 > p.timeout_ns) {
        ok = false;
        atomicOr(p.status, kGruTimeoutGrid);
        break;
      }
    }
    __threadfence();
  }
  tc_fence_before();
  ok = __syncthreads_and(ok) != 0;
  tc_fence_after();

  const int nrows = pl.ntile * B;                                // operand rows (K tile, batch entry) of 128 bytes
  const int ngroups = (nrows + 32 * kLoadsPerGroup - 1) / (32 * kLoadsPerGroup);

  if (ok && warp == kWorkers / 32) {
    // ---------------- the warp that issues the MMAs ----------------
    const bool leader = elect_one();
    const uint32_t fmt = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(NB >> 3) << 17);
    const uint32_t idesc0 = fmt | ((uint32_t)(pl.m0 >> 4) << 24), idesc1 = fmt | ((uint32_t)(pl.m1 >> 4) << 24);
    const uint64_t b_desc = operand_desc(x_addr);
    const uint64_t a_desc0 = operand_desc(w_addr);
    const uint64_t a_desc1 = operand_desc(w_addr + (pl.kq - pl.kt0 + kKTile - 1) / kKTile * pl.m0 * 128);
    const uint32_t d0 = tmem, d1 = tmem + NB, a0 = tmem + pl.col0, a1 = a0 + pl.kt0;
    for (int s = 1; ok && s < T; s++) {
      int done_tiles = 0;
      for (int g = 0; ok && g < ngroups; g++) {
        ok = mbar_wait(full_bar + 8 * g, (uint32_t)(s - 1) & 1, 4 * p.timeout_ns, abort_s);
        ok = __all_sync(0xffffffffu, ok) != 0;
        if (!ok) break;
        tc_fence_after();
        const int have = min(kLoadsPerGroup * 32 * (g + 1), nrows) / B;
        if (leader) {
          for (int kt = done_tiles; kt < have; kt++) {
            const int steps = min(4, (pl.kq - kt * kKTile) / 8);
            const uint64_t b = b_desc + (uint64_t)(kt * NB * 128 >> 4);
            const int k0 = kt * kKTile;
            if (k0 < pl.kt0) {
#pragma unroll
              for (int ks = 0; ks < 4; ks++)
                if (ks < steps) tc_mma_ts(d0, a0 + k0 + 8 * ks, b + 2 * ks, idesc0, kt + ks > 0);
            } else {
              const uint64_t a = a_desc0 + (uint64_t)((k0 - pl.kt0) / kKTile * pl.m0 * 128 >> 4);
#pragma unroll
              for (int ks = 0; ks < 4; ks++)
                if (ks < steps) tc_mma_ss(d0, a + 2 * ks, b + 2 * ks, idesc0, kt + ks > 0);
            }
            if (R > 128) {
              if (k0 < pl.kt1) {
#pragma unroll
                for (int ks = 0; ks < 4; ks++)
                  if (ks < steps) tc_mma_ts(d1, a1 + k0 + 8 * ks, b + 2 * ks, idesc1, kt + ks > 0);
              } else {
                const uint64_t a = a_desc1 + (uint64_t)((k0 - pl.kt1) / kKTile * pl.m1 * 128 >> 4);
#pragma unroll
                for (int ks = 0; ks < 4; ks++)
                  if (ks < steps) tc_mma_ss(d1, a + 2 * ks, b + 2 * ks, idesc1, kt + ks > 0);
              }
            }
          }
          if (g == ngroups - 1) tc_commit(done_bar);
        }
        done_tiles = have;
        __syncwarp();
      }
    }
    if (!ok && leader) {
      // A wait ran out here or in a worker. Nothing may be in flight when tensor memory is freed.
      *abort_s = 1;
      tc_commit(drain_bar);
      mbar_wait(drain_bar, 0, p.timeout_ns, nullptr);
    }
    __syncwarp();
  } else if (ok) {
    // ---------------- the workers ----------------
    // Worker (u, pk) handles unit u0 + u for the batch entries b0 .. b0 + mine - 1.
    const int u = tid & 15, pk = tid >> 4, b0 = 3 * pk;
    const int mine = pk < npacks ? min(3, B - b0) : 0;
    float carry[3] = {0.f, 0.f, 0.f};   // forward: h_{t-1}; backward: recurrent part of dh_t
    // Operand load `it` of this thread: 16-byte word tid + 256 it of the member's range, i.e. chunk tid % 8 of
    // row tid / 8 + 32 it = (K tile, batch entry). Its place in shared memory, or -1 if there is none:
    const int chunk = tid & 7, row0 = tid >> 3;
    const int last_chunks = (pl.kq - (pl.ntile - 1) * kKTile) / 4;      // valid chunks of the last K tile
    const int inv_b = 65536 / B + 1;                                  // row / B for row < 2048
    auto place = [&](int it) -> int {
      const int row = row0 + 32 * it, kt = (row * inv_b) >> 16, b = row - kt * B;
      return (row < nrows && (kt < pl.ntile - 1 || chunk < last_chunks)) ? (kt * NB + b) * 128 + ((chunk ^ (b & 7)) << 4) : -1;
    };
    const uint32_t* src0 = ring + (size_t)q * ring_member + (size_t)tid * 4;
    constexpr bool two_tiles = R > 128;
    const int quarter = warp & 3, tile = two_tiles ? warp >> 2 : 0, m = tile ? pl.m1 : pl.m0;
    const int r = tile * 128 + (m == 128 ? quarter * 32 + lane : quarter * 16 + (lane & 15));   // row of the accumulator
    const bool row_ok = r < R && (m == 128 || lane < 16);
    const int owner = r / kRows, rr = r % kRows;
    constexpr int kPacks = (NB + 2) / 3, kHalf = (kPacks + 1) / 2;
    // one tile: the first four warps take the first half of the packs, the others the rest
    const int pk_lo = two_tiles || warp < 4 ? 0 : kHalf, pk_hi = min(npacks, two_tiles || warp >= 4 ? kPacks : kHalf);
    uint4* xout = p.xchg + (((size_t)dir * nblocks + grp * C + owner) * C + q) * 2 * xslot + rr;
    const bool stamping = p.prof && tid == 0 && blockIdx.x == 0 && blockIdx.y == 0;
    auto stamp = [&](int s, int i) {
      if (stamping) p.prof[(size_t)s * 8 + i] = gtimer();
    };
    auto give_up = [&](uint32_t why) {
      atomicOr(p.status, why);
      *abort_s = 1;
      return false;
    };

    // One recurrent product: the operand words tagged `tag`, the MMAs, the exchange inside the group.
    // acc[g][j] receives the sum of this thread's unit (forward: gate g) for batch entry b0 + j.
    // `good` falls when one of this thread's waits has run out; every worker comes through workers_sync_and() all the
    // same, where all of them learn of it (the result is false then).
    auto product = [&](uint32_t tag, int s, float (*acc)[3], bool& good) -> bool {
      const uint32_t parity = (tag - 1) & 1;
      const uint32_t* src = src0 + (size_t)parity * ring_slot;
      constexpr int kSpan = 3;           // groups whose loads are in flight together
      for (int g0 = 0; g0 < ngroups; g0 += kSpan) {
        uint4 v[kSpan * kLoadsPerGroup];
#pragma unroll
        for (int i = 0; i < kSpan * kLoadsPerGroup; i++) {
          const int it = g0 * kLoadsPerGroup + i;
          if (place(it) >= 0) v[i] = ld_words(src + (size_t)it * (kWorkers * 4));
        }
#pragma unroll
        for (int gi = 0; gi < kSpan; gi++) {
          if (g0 + gi < ngroups) {
            uint32_t spins = 0;
            unsigned long long t0 = 0;
            for (;;) {
              bool missing = false;
#pragma unroll
              for (int i = gi * kLoadsPerGroup; i < (gi + 1) * kLoadsPerGroup; i++) {
                const int it = g0 * kLoadsPerGroup + i;
                if (place(it) >= 0 && stale(v[i], tag)) {
                  missing = true;
                  v[i] = ld_words(src + (size_t)it * (kWorkers * 4));
                }
              }
              if (!missing || !good) break;
              if (((++spins) & 63) == 0) {
                const unsigned long long now = gtimer();
                if (t0 == 0) t0 = now;
                if (*abort_s) good = false;
                else if (now - t0 > p.timeout_ns) good = give_up(kGruTimeoutGrid);
              }
            }
#pragma unroll
            for (int i = gi * kLoadsPerGroup; i < (gi + 1) * kLoadsPerGroup; i++) {
              const int at = place(g0 * kLoadsPerGroup + i);
              if (at >= 0) *reinterpret_cast<uint4*>(x_s + at) = v[i];
            }
            fence_proxy_async();
            tc_fence_before();           // this thread's reads of the previous accumulator come before the MMAs
            __syncwarp();
            if (lane == 0) mbar_arrive(full_bar + 8 * (g0 + gi));
          }
        }
      }
      stamp(s, 1);
      if (!mbar_wait(done_bar, parity, 4 * p.timeout_ns, abort_s)) good = *abort_s ? false : give_up(kGruTimeoutMma);
      good = __all_sync(0xffffffffu, good) != 0;
      stamp(s, 2);
      tc_fence_after();
      if (good) {
        uint32_t v[NB + 2];
        v[NB] = v[NB + 1] = 0;
        tc_ld<NB>(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(tile * NB), v);
        if (row_ok) {
          if (owner == q) {
#pragma unroll
            for (int k = 0; k < kPacks; k++)
              if (k >= pk_lo && k < pk_hi)
#pragma unroll
                for (int j = 0; j < 3; j++)
                  if (3 * k + j < NB) own_s[rr * kOwnStride + 3 * k + j] = __uint_as_float(v[3 * k + j]);
          } else {
            uint4* o = xout + (size_t)parity * xslot;
#pragma unroll
            for (int k = 0; k < kPacks; k++)
              if (k >= pk_lo && k < pk_hi) st_pack(o + k * kRows, make_uint4(v[3 * k], v[3 * k + 1], v[3 * k + 2], tag));
          }
        }
      }
      if (!workers_sync_and(good)) return false;
      stamp(s, 3);
      if (mine > 0) {
#pragma unroll
        for (int g = 0; g < kGates; g++)
#pragma unroll
          for (int j = 0; j < 3; j++) acc[g][j] = j < mine ? own_s[(g * kUnits + u) * kOwnStride + b0 + j] : 0.f;
        if (C > 1) {
          const uint4* in = xin + (size_t)parity * xslot + pk * kRows + u;
          // peers one after the other: member q + 1, q + 2, ... of the group
          uint4 v[C > 1 ? C - 1 : 1][kGates];
#pragma unroll
          for (int i = 0; i < C - 1; i++)
#pragma unroll
            for (int g = 0; g < kGates; g++) v[i][g] = ld_pack(in + (size_t)(i < q ? i : i + 1) * 2 * xslot + g * kUnits);
          uint32_t spins = 0;
          unsigned long long t0 = 0;
          for (;;) {
            bool missing = false;
#pragma unroll
            for (int i = 0; i < C - 1; i++)
#pragma unroll
              for (int g = 0; g < kGates; g++)
                if (v[i][g].w != tag) {
                  missing = true;
                  v[i][g] = ld_pack(in + (size_t)(i < q ? i : i + 1) * 2 * xslot + g * kUnits);
                }
            if (!missing || !good) break;
            if (((++spins) & 63) == 0) {
              const unsigned long long now = gtimer();
              if (t0 == 0) t0 = now;
              if (*abort_s) good = false;
              else if (now - t0 > p.timeout_ns) good = give_up(kGruTimeoutGrid);
            }
          }
#pragma unroll
          for (int i = 0; i < C - 1; i++)
#pragma unroll
            for (int g = 0; g < kGates; g++) {
              acc[g][0] += __uint_as_float(v[i][g].x);
              acc[g][1] += __uint_as_float(v[i][g].y);
              acc[g][2] += __uint_as_float(v[i][g].z);
            }
        }
      }
      stamp(s, 4);
      return true;
    };

    bool fine = true;    // this thread's waits; a step ends for all workers when one of them has given up
    if (!BWD) {
      const float bias_r = p.b_hh[dir][u0 + u], bias_z = p.b_hh[dir][H + u0 + u], bias_n = p.b_hh[dir][2 * H + u0 + u];
      float gx[3][3];
      auto load_gx = [&](int t) {
#pragma unroll
        for (int j = 0; j < 3; j++)
          if (j < mine) {
            const float* g = p.gx + (((size_t)t * B + b0 + j) * ND + dir) * 3 * H + u0 + u;
            gx[0][j] = __ldg(g); gx[1][j] = __ldg(g + H); gx[2][j] = __ldg(g + 2 * H);
          }
      };
      load_gx(dir ? T - 1 : 0);
      for (int s = 0; s < T; s++) {
        const int t = dir ? T - 1 - s : s;
        float acc[3][3] = {};
        stamp(s, 0);
        if (s > 0 && !product((uint32_t)s, s, acc, fine)) break;
        float4 keep[3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
          if (j < mine) {
            const float hn = bias_n + acc[2][j];
            const float r_ = sigmoidf_(gx[0][j] + (bias_r + acc[0][j]));
            const float z = sigmoidf_(gx[1][j] + (bias_z + acc[1][j]));
            const float n = tanhf(gx[2][j] + r_ * hn);
            carry[j] = n + z * (carry[j] - n);
            keep[j] = make_float4(r_, z, n, hn);
          }
        }
        if (s + 1 < T) {
          uint32_t* o = ring + (size_t)(s & 1) * ring_slot;
#pragma unroll
          for (int j = 0; j < 3; j++)
            if (j < mine) st_word(o + ring_at(0, u, b0 + j), tagged(carry[j], (uint32_t)s + 1));
        }
        stamp(s, 5);
        // The peers do not wait for what follows.
#pragma unroll
        for (int j = 0; j < 3; j++)
          if (j < mine) {
            p.y[((size_t)t * B + b0 + j) * (ND * H) + dir * H + u0 + u] = carry[j];
            if (p.rsv) p.rsv[((size_t)(dir * T + t) * B + b0 + j) * H + u0 + u] = keep[j];
          }
        if (s + 1 < T) load_gx(dir ? T - 2 - s : s + 1);
      }
    } else {
      BwdInputs in;
      float sum[4] = {0.f, 0.f, 0.f, 0.f}, part[4] = {0.f, 0.f, 0.f, 0.f};   // bias gradients, in runs of 16 steps
      load_bwd_inputs(p, in, dir ? 0 : T - 1, dir, u0 + u, b0, mine);
      for (int s = 0; s < T; s++) {
        const int t = dir ? s : T - 1 - s;
        float keep[3], g[4][3];
        stamp(s, 0);
#pragma unroll
        for (int j = 0; j < 3; j++) {
          keep[j] = 0.f;
          if (j < mine) {
            const float r_ = in.a[j].x, z = in.a[j].y, n = in.a[j].z, hn = in.a[j].w;
            const float dh = in.dy[j] + carry[j];
            const float dn = dh * (1.f - z) * (1.f - n * n);
            g[0][j] = dn * hn * r_ * (1.f - r_);
            g[1][j] = dh * (in.hp[j] - n) * z * (1.f - z);
            g[2][j] = dn;
            g[3][j] = dn * r_;
            keep[j] = dh * z;
          }
        }
        if (s + 1 < T) {
          uint32_t* o = ring + (size_t)(s & 1) * ring_slot;
#pragma unroll
          for (int k = 0; k < 3; k++)
#pragma unroll
            for (int j = 0; j < 3; j++)
              if (j < mine) st_word(o + ring_at(k, u, b0 + j), tagged(g[k == 2 ? 3 : k][j], (uint32_t)s + 1));
        }
        stamp(s, 5);
        // The peers do not wait for what follows.
#pragma unroll
        for (int j = 0; j < 3; j++)
          if (j < mine) {
            float* o = p.dg + ((size_t)t * B + b0 + j) * (ND * 4 * H) + u0 + u;
#pragma unroll
            for (int k = 0; k < 3; k++) o[(dir * 3 + k) * H] = g[k][j];
            o[(ND * 3 + dir) * H] = g[3][j];
#pragma unroll
            for (int k = 0; k < 4; k++) part[k] += g[k][j];
          }
        if ((s & 15) == 15) {
#pragma unroll
          for (int k = 0; k < 4; k++) { sum[k] += part[k]; part[k] = 0.f; }
        }
        if (s + 1 < T) {
          load_bwd_inputs(p, in, dir ? s + 1 : T - 2 - s, dir, u0 + u, b0, mine);
          float acc[1][3] = {};
          if (!product((uint32_t)s + 1, s, acc, fine)) break;
#pragma unroll
          for (int j = 0; j < 3; j++) carry[j] = keep[j] + acc[0][j];
        }
      }
      // Bias gradients of this block's units. The operand area is free: every MMA has been waited for.
      float* red = reinterpret_cast<float*>(x_s);
      if (mine > 0)
#pragma unroll
        for (int k = 0; k < 4; k++) red[(pk * 4 + k) * kUnits + u] = sum[k] + part[k];
      workers_sync_and(true);
      if (tid < 4 * kUnits) {
        float v = 0.f;
        for (int i = 0; i < npacks; i++) v += red[i * 4 * kUnits + tid];
        const int k = tid / kUnits;
        float* o = p.db + dir * 6 * H + u0 + tid % kUnits;
        if (k != 3) o[k * H] = v;               // dr, dz, dn
        if (k != 2) o[(k == 3 ? 5 : k + 3) * H] = v;   // dr, dz, dn * r
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kWorkers / 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)kTmemCols) : "memory");
}

// ---- host side ------------------------------------------------------------------------------

unsigned long long* g_prof = nullptr;   // set by gru_persistent_set_profile()

bool dims_ok(const GruDims& d) {
  return d.T >= 1 && d.T < 4096 && d.B >= 1 && d.B <= 32 && d.H >= 128 && d.H <= 1024 && d.H % 128 == 0 && (d.ndir == 1 || d.ndir == 2);
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

int mma_n(const GruDims& d) { return d.B <= 16 ? 16 : 32; }

int choose_split(const GruDims& d, bool bwd) {
  if (const char* e = getenv(bwd ? "GRU_CB" : "GRU_CF")) return atoi(e);
  return bwd ? 8 : 4;
}

// Bytes of partial sums (fp32, 32 batch rows, a block's own included) that a step exchanges with the
// widest groups that the dimensions allow: 4 blocks forward, 16 backward.
size_t exchange_bytes(const GruDims& d) {
  const size_t blocks = (size_t)d.ndir * (d.H / kUnits);
  const int widest = d.H / kUnits % 16 == 0 ? 16 : 8;
  return blocks * 32 * 4 * std::max(4 * RowsPerOwner<false>::value, widest * RowsPerOwner<true>::value);
}
constexpr size_t kSyncBytes = 1024;
// Both slots of the ring. The backward pass is the larger one: three words per unit and batch entry, and the last K tile of
// a member may be half empty.
size_t ring_bytes(const GruDims& d) { return (size_t)d.ndir * 2 * (3 * d.H + 16 * 16) * 32 * 4; }

template <bool BWD, int C, int NB>
cudaError_t launch_as(const Params& p, cudaStream_t stream) {
  const GruDims& d = p.d;
  const Plan pl = make_plan<BWD>(C, NB, d.H);
  auto kernel = gru_persistent_kernel<BWD, C, NB>;
  const int smem = std::max(pl.smem(), kMinSmem);
  dim3 grid(d.H / kUnits, d.ndir), block(kThreads);
  if (grid.x > (unsigned)kMaxBlocksPerDir || grid.x % C != 0 || pl.ntile > 4 * kMaxGroups) return cudaErrorInvalidValue;
  // The attribute belongs to a device: set once for each, to all that a block can have.
  static std::atomic<uint64_t> granted{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 64 || !(granted.load(std::memory_order_relaxed) >> dev & 1)) {
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024)) != cudaSuccess) return e;
    if (dev < 64) granted.fetch_or(1ull << dev, std::memory_order_relaxed);
  }
  void* args[] = {(void*)&p};
  return cudaLaunchCooperativeKernel((const void*)kernel, grid, block, args, (size_t)smem, stream);
}

template <bool BWD, int NB>
cudaError_t launch_split(int c, const Params& p, cudaStream_t stream) {
  switch (c) {
    case 1: return launch_as<BWD, 1, NB>(p, stream);
    case 2: return launch_as<BWD, 2, NB>(p, stream);
    case 4: return launch_as<BWD, 4, NB>(p, stream);
    case 8: if (BWD) return launch_as<BWD, BWD ? 8 : 1, NB>(p, stream); break;
    case 16: if (BWD) return launch_as<BWD, BWD ? 16 : 1, NB>(p, stream); break;
  }
  return cudaErrorInvalidValue;
}

template <bool BWD>
cudaError_t launch(Params& p, void* scratch, double timeout_s, cudaStream_t stream) {
  char* w = (char*)scratch;
  p.sync = (uint32_t*)w;
  p.ring = (uint32_t*)(w + kSyncBytes);
  p.xchg = (uint4*)(w + kSyncBytes + ring_bytes(p.d));
  p.timeout_ns = (unsigned long long)(timeout_s * 1e9);
  p.prof = g_prof;
  const int c = choose_split(p.d, BWD);
  return mma_n(p.d) == 16 ? launch_split<BWD, 16>(c, p, stream) : launch_split<BWD, 32>(c, p, stream);
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

// Both slots of the exchange area hold three partial sums per 16 bytes, rounded up to whole 16-byte words per row: 11 for
// 32 batch entries, less than 3/2 of the plain size.
size_t gru_persistent_scratch_bytes(const GruDims& d) { return dims_ok(d) ? kSyncBytes + ring_bytes(d) + 3 * exchange_bytes(d) : 0; }

cudaError_t gru_persistent_forward(const GruDims& d, const float* const* w_hh, const float* const* b_hh, const float* gx, float* y,
                                   float* rsv, void* scratch, uint32_t* status, double timeout_s, cudaStream_t stream) {
  if (!dims_ok(d) || !aligned16(rsv) || !aligned16(scratch)) return cudaErrorInvalidValue;
  Params p{};
  p.d = d;
  for (int i = 0; i < d.ndir; i++) {
    if (!aligned16(w_hh[i])) return cudaErrorInvalidValue;
    p.w_hh[i] = w_hh[i];
    p.b_hh[i] = b_hh[i];
  }
  p.gx = gx;
  p.y = y;
  p.rsv = (float4*)rsv;
  p.status = status;
  return launch<false>(p, scratch, timeout_s, stream);
}

cudaError_t gru_persistent_backward(const GruDims& d, const float* const* w_hh, const float* y, const float* rsv, const float* dy,
                                    float* dg, float* db, void* scratch, uint32_t* status, double timeout_s, cudaStream_t stream) {
  if (!dims_ok(d) || !aligned16(rsv) || !aligned16(scratch)) return cudaErrorInvalidValue;
  Params p{};
  p.d = d;
  for (int i = 0; i < d.ndir; i++) {
    if (!aligned16(w_hh[i])) return cudaErrorInvalidValue;
    p.w_hh[i] = w_hh[i];
  }
  p.y = const_cast<float*>(y);
  p.rsv = (float4*)const_cast<float*>(rsv);
  p.dy = dy;
  p.dg = dg;
  p.db = db;
  p.status = status;
  return launch<true>(p, scratch, timeout_s, stream);
}

}  // namespace gpu
}  // namespace bc

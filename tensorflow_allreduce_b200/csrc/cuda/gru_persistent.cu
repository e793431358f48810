// Persistent bidirectional GRU layer for sm_100a (see gru_persistent.h for the interface): backward pass and host side. The forward
// pass is in gru_forward.cu.
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
//   * Lines that another SM has just written are slow to read: 128 blocks that read 32 KB each take 1130 cycles
//     when nothing was written, 1406 (the last block 1863) when it was. That is why the volume per block matters,
//     why a loader thread reads 32 bytes per request, and why nothing is polled before it can be there.
//   * Operand A from tensor memory: one M = 128, N = 32, K = 8 instruction takes 20 cycles, from shared
//     memory 45 (it reads 5 KiB at 128 B per cycle). Weights that do not fit in the 512 columns stay in
//     shared memory (forward pairs at H = 1024: 32 of 512 columns).
//   * The MMAs are issued by an elected lane of a warp of its own; issued from under a
//     `threadIdx.x == n` branch the same M = 64, N = 32 instruction took 55 cycles instead of 26. With two warps per
//     scheduler every instruction of a serial chain costs four to six cycles, so the loops are kept short.
//   * Two chains of half the batch each, meant to hide one's waits behind the other's work, were slower (4.7 us per step
//     forward where one chain took 3.8): what bounds the exchange is the fresh lines, not the number of bytes in flight.
// Microseconds per step: see choose_split(). The variants that the comments of this file compare were measured with the code as it
// stands, other figures of a variant that is not here any more beside the time that the kernel took then.
//
// Every wait is bounded by %globaltimer. When a wait runs out the block records a status bit, goes through its remaining steps without
// waiting, and like every block waits (bounded) for its own MMAs in flight before it frees its tensor memory and returns.
#include "gru_common.cuh"

#include <algorithm>
#include <atomic>

namespace bc {
namespace gpu {

namespace {

using namespace gru;

constexpr int kKTile = 32;            // fp32 elements in one 128-byte swizzle row
constexpr int kGateThreads = 256;     // eight warps: accumulator read-back, exchange, gate math
constexpr int kLoadThreads = 256;     // eight warps: poll the operand words and put them into shared memory
constexpr int kThreads = kGateThreads + kLoadThreads + 32;   // and the warp that issues the MMAs
constexpr int kMaxBlocksPerDir = 64;  // H / 16 at H = 1024
constexpr int kLoadBytes = kLoadThreads * 32;   // operand bytes that one load of every loader thread brings
constexpr int kMaxGroups = 8;         // pipeline groups (one mbarrier each) of a step: 32 K tiles of 32 batch rows in pairs of loads
// ---- PTX wrappers beside those of tcgen05_prims.cuh ---------------------------------------------

// N consecutive columns of this thread's tensor-memory lane: the packs that one warp reads back (see `send` below).
template <int N> __device__ __forceinline__ void tc_ld(uint32_t taddr, uint32_t* r);
template <> __device__ __forceinline__ void tc_ld<6>(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%6];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x2.b32 {%4, %5}, [%7];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5])
      : "r"(taddr), "r"(taddr + 4) : "memory");
}
template <> __device__ __forceinline__ void tc_ld<9>(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%9];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x1.b32 {%8}, [%10];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8])
      : "r"(taddr), "r"(taddr + 8) : "memory");
}
// Words that travel between blocks.
__device__ __forceinline__ void st_word(uint32_t* p, uint32_t v) { asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
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
__device__ __forceinline__ bool stale(const Words& v, uint32_t tag) {
  uint32_t d = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) d |= v.w[i] ^ tag;
  return (d & kTagMask) != 0;
}

// Barrier 1: all gate and loader warps have read the accumulator and sent their part of it; the loaders only arrive. It has no limit, and
// a warp that arrived twice before the others have come once would complete it without them and leave them waiting for good. So gate and
// loader warps come to it once per step whatever waits have run out, and the loaders never before the gate warps have passed it the last
// time: their wait for the block's publication is the one that is never skipped or cut short.
__device__ __forceinline__ void sent_sync() { asm volatile("barrier.cta.sync 1, 512;" ::: "memory"); }
__device__ __forceinline__ void sent_arrive() { asm volatile("barrier.cta.arrive 1, 512;" ::: "memory"); }
__device__ __forceinline__ void gates_sync() { asm volatile("barrier.cta.sync 2, 256;" ::: "memory"); }

// Where everything of one block lives; a function of the pass, the split and the dimensions.
struct Plan {
  int kq;            // K range of a member: columns of the recurrent weights it holds
  int ntile;         // K tiles of 32 (the last one may be half)
  int m;             // M of the MMAs: rows of the group, padded to 64 or 128
  int k_tmem;        // K columns that live in tensor memory; the others live in shared memory
  int x_bytes, w_bytes, own_bytes;
  __host__ __device__ int smem() const { return 1024 + x_bytes + w_bytes + own_bytes + 256; }
};
__host__ __device__ constexpr int packs_of(int batch) { return (batch + 2) / 3; }   // three partial sums and the step number per 16 bytes

__host__ __device__ inline Plan make_plan(int C, int nb, int H) {
  Plan p;
  const int rows = kUnits * C;
  p.kq = 3 * H / C;
  p.ntile = (p.kq + kKTile - 1) / kKTile;
  p.m = rows > 64 ? 128 : 64;
  const int room = (int)kTmemCols - nb;                 // the accumulator takes the first nb columns
  p.k_tmem = p.kq <= room ? p.kq : room / kKTile * kKTile;
  p.x_bytes = p.ntile * nb * 128;
  p.w_bytes = (p.kq - p.k_tmem + kKTile - 1) / kKTile * p.m * 128;
  p.own_bytes = kUnits * packs_of(nb) * 16;
  return p;
}

// The 16 weights of row `r` of the group at columns k0 .. k0 + 15 of member q's K range (k0 a multiple of 16).
// Rows ordered owner, unit; K ordered gate, unit of the range   W[g * H + unit'][unit]
// A run of 16 columns stays inside one gate, because a member's range of units is a multiple of 16.
__device__ __forceinline__ void load_weights16(const float* w, int H, int C, int grp, int q, int r, int k0, float* o) {
  const int range = H / C, g = k0 / range, kk = q * range + k0 - g * range;
  const float* p = w + (size_t)(g * H + kk) * H + grp * C * kUnits + r;
#pragma unroll
  for (int i = 0; i < 16; i++) o[i] = __ldg(p + (size_t)i * H);
}

// C: blocks per group; NB: N of the MMA (16 or 32, at least the batch); kLoadsPerGroup: loads of a loader thread per
// pipeline group. With five loads or more, groups of four, one in flight, win (us per step, B = 32: H = 1024 forward 3.80 -> 3.68, backward
// 4.43 -> 4.24, H = 512 backward 4.07 -> 3.39: fewer polls of words that are not there yet; H = 768 forward loses, 3.23 -> 3.31); with fewer,
// pairs do (forward H = 512, B = 32: 2.80 against 2.91, B = 8: 2.24 against 2.51).
//
// Three kinds of warps, so that no work off the chain of a step (output stores, prefetches) delays the next
// product: gate warps, loader warps, and one warp that issues the MMAs. One barrier each says that
// the operand is in shared memory (full[group]: loaders -> MMA), that the accumulator is complete (done:
// MMA -> all), that it has been read (read: all -> MMA), and that this block has published (published: gates -> loaders).
template <int C, int NB, int kLoadsPerGroup>
__global__ void __launch_bounds__(kThreads, 1) gru_backward_kernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);

  constexpr int kRows = kUnits;            // accumulator rows of a member
  constexpr int R = kRows * C;
  constexpr int kGates = 1;                // accumulator rows per unit
  constexpr int kGateWords = 3;            // operand words that a (unit, batch) pair publishes per step
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int dir = blockIdx.y, u0 = blockIdx.x * kUnits;
  const int T = p.d.T, B = p.d.B, H = p.d.H, ND = p.d.ndir;
  const int nblocks = gridDim.x;
  const int grp = blockIdx.x / C, q = blockIdx.x % C;
  const Plan pl = make_plan(C, NB, H);
  const int npacks = packs_of(B);

  uint8_t* x_s = smem;
  uint8_t* w_s = smem + pl.x_bytes;
  uint4* own_s = reinterpret_cast<uint4*>(w_s + pl.w_bytes);                       // this block's own partial sums: [pack][row]
  uint64_t* bar_s = reinterpret_cast<uint64_t*>(w_s + pl.w_bytes + pl.own_bytes);  // full[kMaxGroups], done, drain, read, published
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_s + kMaxGroups + 4);
  volatile int* abort_s = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t full_bar = smem_u32(bar_s), done_bar = full_bar + 8 * kMaxGroups, drain_bar = done_bar + 8, read_bar = done_bar + 16, pub_bar = done_bar + 24;
  const uint32_t x_addr = smem_u32(x_s), w_addr = smem_u32(w_s);

  if (tid == 0) {
    for (int i = 0; i < kMaxGroups; i++) mbar_init(full_bar + 8 * i, kLoadThreads / 32);
    mbar_init(done_bar, 1);
    mbar_init(drain_bar, 1);
    mbar_init(read_bar, (kGateThreads + kLoadThreads) / 32);
    mbar_init(pub_bar, kGateThreads / 32);
    *abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kThreads / 32 - 1) {
    tmem_alloc(tmem_slot, kTmemCols);
  }

  // The part of the ring that this block writes (both slots) and the partial sums that it will
  // receive: cleared, so that nothing of an earlier launch passes for a word of this one.
  const int range = H / C;                                       // units of one member's K range
  const uint32_t ring_member = (uint32_t)pl.ntile * NB * kKTile;  // words of one member's range and slot
  const uint32_t ring_slot = ring_member * C;
  uint32_t* ring = p.ring + (size_t)dir * 2 * ring_slot;
  // word of (gate g, unit u0 + u, batch b): member u0 / range, column g * range + u0 % range + u
  const uint32_t my_member = (uint32_t)(u0 / range) * ring_member;
  const int my_col = u0 % range;
  auto ring_at = [&](int g, int u, int b) -> uint32_t {
    const int k = g * range + my_col + u;
    return my_member + (uint32_t)((k >> 5) * NB + b) * kKTile + (k & 31);
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

  // The group's weight rows for this block's K range, resident for the whole sequence. With M = 128 row r is
  // lane r of tensor memory; with M = 64 it is lane (r / 16) * 32 + r % 16, the other lanes are not used.
  const float* w = p.w_hh[dir];
  const int quarter = warp & 3;
  const int lane_row = pl.m == 128 ? quarter * 32 + lane : quarter * 16 + (lane & 15);
  const bool row_ok = lane_row < R && (pl.m == 128 || lane < 16);
  if (warp < 8) {
    for (int k0 = 16 * (warp >> 2); k0 < pl.k_tmem; k0 += 32) {
      float v[16];
#pragma unroll
      for (int i = 0; i < 16; i++) v[i] = 0.f;
      if (row_ok) load_weights16(w, H, C, grp, q, lane_row, k0, v);
      __syncwarp();
      tmem_st16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(NB + k0), v);
    }
    tmem_st_wait();
    for (int i = tid; i < pl.m * ((pl.kq - pl.k_tmem) / 16); i += 256) {
      const int r = i % pl.m, k = (i / pl.m) * 16;                     // counted from k_tmem
      float v[16];
#pragma unroll
      for (int e = 0; e < 16; e++) v[e] = 0.f;
      if (r < R) load_weights16(w, H, C, grp, q, r, pl.k_tmem + k, v);
      uint8_t* row = w_s + ((k >> 5) * pl.m + r) * 128;
#pragma unroll
      for (int e = 0; e < 4; e++)
        reinterpret_cast<float4*>(row)[(((k & 31) >> 2) + e) ^ (r & 7)] = make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
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

  // A loader thread's load `it` is the 32-byte word lt + 256 it of the member's range, i.e. chunks 2 (lt % 4) and the next
  // of batch row lt / 4 % NB in K tile it * (64 / NB) + lt / 4 / NB: 8 KiB further per load in the ring and in shared memory.
  constexpr int kTilesPerLoad = 64 / NB;
  const int nloads = (pl.ntile + kTilesPerLoad - 1) / kTilesPerLoad;
  const int ngroups = (nloads + kLoadsPerGroup - 1) / kLoadsPerGroup;
  auto give_up = [&](uint32_t why) {
    atomicOr(p.status, why);
    *abort_s = 1;
    return false;
  };

  // Read-back of the accumulator, by gate and loader warps together: a warp may read the quarter warp % 4 of the lanes, and
  // the four warps of a quarter share the packs of its rows (three batch entries each).
  constexpr int kPacks = packs_of(NB), kPart = (kPacks + 3) / 4;
  const int owner = lane_row / kRows, rr = lane_row % kRows;
  const int pk_lo = (warp >> 2) * kPart, pk_n = max(0, min(kPart, npacks - pk_lo));
  uint4* xout = p.xchg + (((size_t)dir * nblocks + grp * C + owner) * C + q) * 2 * xslot + pk_lo * kRows + rr;
  auto send = [&](uint32_t tag, uint32_t parity) {
    uint32_t v[3 * kPart];
    tc_fence_after();
    // a few columns past the accumulator's are read as well (they are inside the allocation) and sent as padding
    tc_ld<3 * kPart>(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(3 * pk_lo), v);
    tc_fence_before();
    if (lane == 0) mbar_arrive(read_bar);
    if (row_ok) {
      if (owner == q) {
#pragma unroll
        for (int i = 0; i < kPart; i++)
          if (i < pk_n) own_s[(pk_lo + i) * kRows + rr] = make_uint4(v[3 * i], v[3 * i + 1], v[3 * i + 2], 0);
      } else {
        uint4* o = xout + (parity ? xslot : 0);
#pragma unroll
        for (int i = 0; i < kPart; i++)
          if (i < pk_n) st_pack(o + i * kRows, make_uint4(v[3 * i], v[3 * i + 1], v[3 * i + 2], tag));
      }
    }
  };

  if (ok && warp == kThreads / 32 - 1) {
    // ---------------- the warp that issues the MMAs ----------------
    const bool leader = elect_one();
    const uint32_t fmt = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(NB >> 3) << 17);
    const uint32_t idesc = fmt | ((uint32_t)(pl.m >> 4) << 24);
    const uint64_t b_desc = operand_desc(x_addr), a_desc = operand_desc(w_addr);
    const uint32_t a_tmem = tmem + NB;
    const int full_tiles = pl.kq / kKTile;              // and perhaps half a tile behind them
    const int ts = pl.k_tmem / kKTile;                  // full K tiles whose weights are in tensor memory
    constexpr uint32_t kBStep = NB * 128 / 16;          // descriptor units from one K tile to the next
    const uint32_t a_step = (uint32_t)pl.m * 128 / 16;
    for (int s = 1; ok && s < T; s++) {
      if (s > 1) ok = mbar_wait(read_bar, (uint32_t)s & 1, 4 * p.timeout_ns, abort_s);
      for (int g = 0; g < ngroups; g++) {
        ok = ok && mbar_wait(full_bar + 8 * g, (uint32_t)(s - 1) & 1, 4 * p.timeout_ns, abort_s);
        ok = __all_sync(0xffffffffu, ok) != 0;
        if (!ok) break;
        tc_fence_after();
        if (leader) {
          const int lo = g * kLoadsPerGroup * kTilesPerLoad, hi = min(full_tiles, lo + kLoadsPerGroup * kTilesPerLoad);
          uint64_t b = b_desc + (uint64_t)((uint32_t)lo * kBStep);
          uint32_t acc = lo > 0, a = a_tmem + lo * kKTile;
          int kt = lo;
#pragma unroll 2
          for (; kt < min(hi, ts); kt++) {
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
              tc_mma_ts(tmem, a + 8 * ks, b + 2 * ks, idesc, acc);
              acc = 1;
            }
            a += kKTile;
            b += kBStep;
          }
          uint64_t as = a_desc + (uint64_t)((uint32_t)max(0, kt - ts) * a_step);
          for (; kt < hi; kt++) {
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
              tc_mma_ss(tmem, as + 2 * ks, b + 2 * ks, idesc, acc);
              acc = 1;
            }
            as += a_step;
            b += kBStep;
          }
          if (g == ngroups - 1) {
            if (full_tiles < pl.ntile) {
#pragma unroll
              for (int ks = 0; ks < 2; ks++) {
                if (full_tiles * kKTile < pl.k_tmem) tc_mma_ts(tmem, a_tmem + full_tiles * kKTile + 8 * ks, b + 2 * ks, idesc, full_tiles + ks > 0);
                else tc_mma_ss(tmem, as + 2 * ks, b + 2 * ks, idesc, full_tiles + ks > 0);
              }
            }
            tc_commit(done_bar);
          }
        }
        __syncwarp();
      }
    }
    if (leader) {
      if (!ok && !*abort_s) give_up(kGruTimeoutBlock);
      // Nothing may be in flight when tensor memory is freed, whatever this or another warp has not waited for.
      tc_commit(drain_bar);
      mbar_drain(drain_bar, 0);
    }
    __syncwarp();
  } else if (ok && warp >= kGateThreads / 32) {
    // ---------------- loaders ----------------
    const int lt = tid - kGateThreads, chunk = 2 * (lt & 3), row = lt >> 2, b = row & (NB - 1), kt0 = row / NB;
    const int last_chunks = (pl.kq - (pl.ntile - 1) * kKTile) / 4;      // valid chunks of the last K tile
    const uint32_t dst = x_addr + (uint32_t)(row * 128 + ((chunk ^ (b & 7)) << 4));
    const uint32_t* src0 = ring + (size_t)q * ring_member + (size_t)lt * 8;
    // loads of this thread: K tiles kt0, kt0 + kTilesPerLoad, ... below ntile, the last one only if it has these chunks
    const int tiles_mine = chunk < last_chunks ? pl.ntile : pl.ntile - 1;
    const int mine = b < B && kt0 < tiles_mine ? (tiles_mine - kt0 + kTilesPerLoad - 1) / kTilesPerLoad : 0;
    // Cycles from a block's own publication to its first poll: about what the operand words of a step take to arrive, but
    // not so little that polls meet the partial sums of groups that are still exchanging them, and not so much that this block is the
    // last one. 80 bytes per cycle out of 55 to 160 tried; nothing to exchange: C = 1. No pause / `read` alone / this rule, us per step: forward
    // H = 1024 B = 32 3.99 / 3.74 / 3.68, B = 8 3.00 / 2.88 / 2.78, B = 1 2.97 / 2.92 / 2.59, H = 256 B = 32 2.34 / 2.27 / 2.19;
    // backward H = 1024 B = 1 2.97 / 2.91 / 2.82. Of 36 passes (H = 128 to 1024, B = 1, 8, 32) none is slower than with `read` alone by
    // more than 1.3 %; those of H = 128 would be up to 5 % faster without a pause.
    const uint32_t read = (uint32_t)(pl.ntile * B * 128) / 80;
    const uint32_t pause = C == 1 ? read / 2 : C == 2 ? min(max(read, 300u), 600u) : C == 4 ? min(read, 300u) : max(read, (uint32_t)p.d.H / 3);
    constexpr int kSpan = kLoadsPerGroup == 4 ? 1 : 3;           // groups whose loads are in flight together
    bool good = true;
    // Every step is gone through to the end even when a wait has run out; the waits then end at once, but for the first.
    for (int s = 1; s < T; s++) {
      const uint32_t tag = (uint32_t)s, parity = (uint32_t)(s - 1) & 1;
      const uint32_t* src = src0 + (size_t)parity * ring_slot;
      // Not before this block has published its own words of the step, and then only when the others' are about to
      // arrive: polling takes L2 bandwidth from the blocks that still exchange partial sums. (Backward, H = 1024, B = 32:
      // from the publication on 4.45 us per step, with the pause 4.24; polling all the time took 6.8 where these took 4.75 and 4.4.)
      // The gate warps always get there: of their waits before it each runs out once, five limits in all.
      if (!mbar_wait(pub_bar, parity, 16 * p.timeout_ns + 1000000000ull, nullptr)) good = give_up(kGruTimeoutBlock);
      for (const uint32_t c0 = clock32(); clock32() - c0 < pause;) {
      }
      for (int g0 = 0; g0 < ngroups; g0 += kSpan) {
        Words v[kSpan * kLoadsPerGroup];
#pragma unroll
        for (int i = 0; i < kSpan * kLoadsPerGroup; i++)
          if (g0 * kLoadsPerGroup + i < mine) ld_words(src + (g0 * kLoadsPerGroup + i) * (kLoadBytes / 4), v[i]);
#pragma unroll
        for (int gi = 0; gi < kSpan; gi++) {
          if (g0 + gi < ngroups) {
            uint32_t spins = 0;
            unsigned long long t0 = 0;
            for (;;) {
              bool missing = false;
#pragma unroll
              for (int i = gi * kLoadsPerGroup; i < (gi + 1) * kLoadsPerGroup; i++) {
                if (g0 * kLoadsPerGroup + i < mine && stale(v[i], tag)) {
                  missing = true;
                  ld_words(src + (g0 * kLoadsPerGroup + i) * (kLoadBytes / 4), v[i]);
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
            for (int i = gi * kLoadsPerGroup; i < (gi + 1) * kLoadsPerGroup; i++)
              if (g0 * kLoadsPerGroup + i < mine)
                st_shared2(dst + (g0 * kLoadsPerGroup + i) * kLoadBytes, v[i]);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(full_bar + 8 * (g0 + gi));
          }
        }
      }
      // The MMAs have read the operand area and written the accumulator.
      if (good && !mbar_wait(done_bar, parity, 4 * p.timeout_ns, abort_s)) good = *abort_s ? false : give_up(kGruTimeoutMma);
      if (__all_sync(0xffffffffu, good)) send(tag, parity);
      else good = false;
      sent_arrive();
    }
  } else if (ok) {
    // ---------------- gates ----------------
    // Thread (u, pk) handles unit u0 + u for the batch entries b0 .. b0 + mine - 1.
    const int u = tid & 15, pk = tid >> 4, b0 = 3 * pk;
    const int mine = pk < npacks ? min(3, B - b0) : 0;
    float carry[3] = {0.f, 0.f, 0.f};   // forward: h_{t-1}; backward: recurrent part of dh_t
    const uint4* xmine = xin + pk * kRows + u;
    const uint4* own_mine = own_s + pk * kRows + u;
    const bool stamping = p.prof && tid == 0 && blockIdx.x == 0 && blockIdx.y == 0;
    auto stamp = [&](int s, int i) {
      if (stamping) p.prof[(size_t)s * 8 + i] = gtimer();
    };

    // One recurrent product, number k = 0, 1, ...: wait for the MMAs, exchange inside the group.
    // acc[g][j] receives the sum of this thread's unit (forward: gate g) for batch entry b0 + j.
    // `good` falls when one of this thread's waits has run out; the steps are gone through to the end all the same.
    bool good = true;
    auto product = [&](int k, int s, float (*acc)[3]) {
      const uint32_t tag = (uint32_t)k + 1, parity = (uint32_t)k & 1;
      if (good && !mbar_wait(done_bar, parity, 4 * p.timeout_ns, abort_s)) good = *abort_s ? false : give_up(kGruTimeoutMma);
      stamp(s, 1);
      if (__all_sync(0xffffffffu, good)) send(tag, parity);
      else good = false;
      sent_sync();
      stamp(s, 2);
      if (mine > 0) {
        uint4 v[C > 1 ? C - 1 : 1][kGates];
        const uint4* in = xmine + (parity ? xslot : 0);
        if (C > 1) {
#pragma unroll
          for (int i = 0; i < C - 1; i++)
#pragma unroll
            for (int g = 0; g < kGates; g++) v[i][g] = ld_pack(in + (i < q ? i : i + 1) * 2 * xslot + g * kUnits);
        }
#pragma unroll
        for (int g = 0; g < kGates; g++) {
          const uint4 o = own_mine[g * kUnits];
          acc[g][0] = __uint_as_float(o.x);
          acc[g][1] = __uint_as_float(o.y);
          acc[g][2] = __uint_as_float(o.z);
        }
        if (C > 1) {
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
                  v[i][g] = ld_pack(in + (i < q ? i : i + 1) * 2 * xslot + g * kUnits);
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
      stamp(s, 3);
    };
    // This block's words of a step are on their way: its loaders may begin to poll the others'.
    auto published = [&] {
      __syncwarp();
      if (lane == 0) mbar_arrive(pub_bar);
    };

    const ptrdiff_t step = dir ? 1 : -1;
    const int t_first = dir ? 0 : T - 1;
    const int y_row = ND * H, dg_row = ND * 4 * H;
    const float4* rsv_p = p.rsv + ((size_t)(dir * T + t_first) * B + b0) * H + u0 + u;
    const float* dy_p = p.dy + ((size_t)t_first * B + b0) * y_row + dir * H + u0 + u;
    const float* hp_p = p.y + ((ptrdiff_t)t_first + step) * B * y_row + (ptrdiff_t)b0 * y_row + dir * H + u0 + u;   // h of the step before in the forward pass
    float* dg_p = p.dg + ((size_t)t_first * B + b0) * dg_row + dir * 3 * H + u0 + u;
    const int dnr_off = (ND * 3 - dir * 2) * H;       // from (dir * 3) * H to (ND * 3 + dir) * H
    uint32_t* ring_p[3] = {ring + ring_at(0, u, b0), ring + ring_at(1, u, b0), ring + ring_at(2, u, b0)};
    float4 in_a[3];                                   // r, z, n, W_hn h + b_hn
    float in_hp[3] = {0.f, 0.f, 0.f}, in_dy[3];
    auto load_inputs = [&](bool has_prev) {
#pragma unroll
      for (int j = 0; j < 3; j++)
        if (j < mine) {
          in_a[j] = __ldg(rsv_p + j * H);
          in_dy[j] = __ldg(dy_p + j * y_row);
          in_hp[j] = has_prev ? __ldg(hp_p + j * y_row) : 0.f;
        }
      rsv_p += step * B * H;
      dy_p += step * B * y_row;
      hp_p += step * B * y_row;
    };
    float sum[4] = {0.f, 0.f, 0.f, 0.f}, part[4] = {0.f, 0.f, 0.f, 0.f};   // bias gradients, in runs of 16 steps
    load_inputs(T > 1);
    for (int s = 0; s < T; s++) {
      float keep[3], g[4][3];
      stamp(s, 0);
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const float r_ = in_a[j].x, z = in_a[j].y, n = in_a[j].z, hn = in_a[j].w;
        const float dh = in_dy[j] + carry[j];
        const float dn = dh * (1.f - z) * (1.f - n * n);
        g[0][j] = dn * hn * r_ * (1.f - r_);
        g[1][j] = dh * (in_hp[j] - n) * z * (1.f - z);
        g[2][j] = dn;
        g[3][j] = dn * r_;
        keep[j] = dh * z;
      }
      if (s + 1 < T) {
        const uint32_t slot = (s & 1) ? ring_slot : 0u;
#pragma unroll
        for (int k = 0; k < 3; k++)
#pragma unroll
          for (int j = 0; j < 3; j++)
            if (j < mine) st_word(ring_p[k] + slot + j * kKTile, tagged(g[k == 2 ? 3 : k][j], (uint32_t)s + 1));
        published();
      }
      stamp(s, 4);
      // The peers do not wait for what follows.
#pragma unroll
      for (int j = 0; j < 3; j++)
        if (j < mine) {
          float* o = dg_p + j * dg_row;
#pragma unroll
          for (int k = 0; k < 3; k++) o[k * H] = g[k][j];
          o[dnr_off] = g[3][j];
#pragma unroll
          for (int k = 0; k < 4; k++) part[k] += g[k][j];
        }
      dg_p += step * B * dg_row;
      if ((s & 15) == 15) {
#pragma unroll
        for (int k = 0; k < 4; k++) { sum[k] += part[k]; part[k] = 0.f; }
      }
      if (s + 1 < T) {
        load_inputs(s + 2 < T);
        float acc[1][3] = {};
        product(s, s, acc);
#pragma unroll
        for (int j = 0; j < 3; j++) carry[j] = keep[j] + acc[0][j];
      }
    }
    // Bias gradients of this block's units. The operand area is free: every MMA has been waited for.
    float* red = reinterpret_cast<float*>(x_s);
    if (mine > 0)
#pragma unroll
      for (int k = 0; k < 4; k++) red[(pk * 4 + k) * kUnits + u] = sum[k] + part[k];
    gates_sync();
    if (tid < 4 * kUnits) {
      float v = 0.f;
      for (int i = 0; i < npacks; i++) v += red[i * 4 * kUnits + tid];
      const int k = tid / kUnits;
      float* o = p.db + dir * 6 * H + u0 + tid % kUnits;
      if (k != 3) o[k * H] = v;                        // dr, dz, dn
      if (k != 2) o[(k == 3 ? 5 : k + 3) * H] = v;     // dr, dz, dn * r
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kThreads / 32 - 1)
    tmem_free(tmem, kTmemCols);
}

// ---- host side ------------------------------------------------------------------------------

unsigned long long* g_prof = nullptr;   // set by gru_persistent_set_profile()

bool dims_ok(const GruDims& d) {
  return d.T >= 1 && d.T < 4096 && d.B >= 1 && d.B <= 32 && d.H >= 128 && d.H <= 1024 && d.H % 128 == 0 && (d.ndir == 1 || d.ndir == 2);
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

// Blocks per group. Fewer blocks: more operand words to poll per block and longer MMA chains; more blocks: more partial
// sums, and with one block per group no exchange at all. Microseconds per step (B200, both directions; B = 32 | B = 8; "-": the weights do
// not fit):
//   forward   H   128          256          384          512          768          1024
//     C = 1       1.73 | 1.43  2.19 | 1.71  2.67 | 2.00  2.88 | 2.24  3.84 | 3.12   -   | 3.51
//     C = 2       2.05 | 1.77  2.29 | 1.92  2.64 | 2.07  2.80 | 2.23  3.32 | 2.50  3.68 | 2.78
//   backward
//     C = 2       2.68 | 2.00  3.14 | 2.39  3.84 | 3.53  4.55 | 3.75   -   |  -     -   |  -
//     C = 4       2.31 | 1.88  2.90 | 2.39  3.09 | 2.59  3.40 | 2.81  3.93 | 3.61  4.59 | 4.00
//     C = 8       3.32 | 2.16  3.47 | 2.34  3.64 | 2.63  3.69 | 2.83  4.03 | 3.05  4.24 | 3.21
// The rule misses the best by 0.1 us at most (backward H = 768 B = 32; at B = 1 forward H = 512, 2.17 against 2.07). Wider groups, 4 forward
// and 16 backward, need more rows than one MMA has; they were 0.5 to 1.5 us slower.
// (Both passes took 7.7 us per step at T = 75, B = 3, H = 512 and 9.3 at B = 32, H = 1024 when blocks exchanged through
// counters and TMA and all weights lay in shared memory.)
int choose_split(const GruDims& d, bool bwd) {
  const bool small = d.B <= 16;
  if (bwd) return d.H <= (small ? 256 : 512) ? 4 : 8;
  return d.H <= (small ? 512 : 256) ? 1 : 2;
}

// Bytes of partial sums (fp32, 32 batch rows, a block's own included) of a step with groups of 4 blocks forward and 16 backward, wider
// than any that is launched.
size_t exchange_bytes(const GruDims& d) {
  const size_t blocks = (size_t)d.ndir * (d.H / kUnits);
  const int widest = d.H / kUnits % 16 == 0 ? 16 : 8;
  return blocks * 32 * 4 * std::max(4 * 48, widest * kUnits);
}
constexpr size_t kSyncBytes = 1024;
// Both slots of the ring. The backward pass is the larger one: three words per unit and batch entry, and the last K tile of
// a member may be half empty.
size_t ring_bytes(const GruDims& d) { return (size_t)d.ndir * 2 * (3 * d.H + 16 * 16) * 32 * 4; }

template <int C, int NB, int LPG>
cudaError_t launch_with(const Params& p, cudaStream_t stream) {
  const GruDims& d = p.d;
  const Plan pl = make_plan(C, NB, d.H);
  auto kernel = gru_backward_kernel<C, NB, LPG>;
  const int smem = std::max(pl.smem(), kMinSmem);
  dim3 grid(d.H / kUnits, d.ndir), block(kThreads);
  if (grid.x > (unsigned)kMaxBlocksPerDir || grid.x % C != 0 || (pl.ntile + 64 / NB - 1) / (64 / NB) > LPG * kMaxGroups) return cudaErrorInvalidValue;
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

template <int C, int NB>
cudaError_t launch_as(const Params& p, cudaStream_t stream) {
  const int loads = (make_plan(C, NB, p.d.H).ntile + 64 / NB - 1) / (64 / NB);
  return loads >= 5 ? launch_with<C, NB, 4>(p, stream) : launch_with<C, NB, 2>(p, stream);
}

void fill(Params& p, void* scratch, double timeout_s) {
  char* w = (char*)scratch;
  p.sync = (uint32_t*)w;
  p.ring = (uint32_t*)(w + kSyncBytes);
  p.xchg = (uint4*)(w + kSyncBytes + ring_bytes(p.d));
  p.timeout_ns = (unsigned long long)(timeout_s * 1e9);
  p.prof = g_prof;
}

cudaError_t launch_backward(const Params& p, cudaStream_t stream) {
  const bool wide = choose_split(p.d, true) > 4;
  if (p.d.B <= 16) return wide ? launch_as<8, 16>(p, stream) : launch_as<4, 16>(p, stream);
  return wide ? launch_as<8, 32>(p, stream) : launch_as<4, 32>(p, stream);
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

// Behind the ring every block has two slots of partial sums, three per 16 bytes, from every member of its group in the wider of the two
// passes (its own stay in shared memory; their place is not used).
size_t gru_persistent_scratch_bytes(const GruDims& d) {
  if (!dims_ok(d)) return 0;
  const size_t rows = std::max(choose_split(d, false) * 48, choose_split(d, true) * kUnits);
  return kSyncBytes + ring_bytes(d) + (size_t)d.ndir * (d.H / kUnits) * 2 * packs_of(d.B) * rows * 16;
}

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
  fill(p, scratch, timeout_s);
  return launch_forward(p, stream);
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
  fill(p, scratch, timeout_s);
  return launch_backward(p, stream);
}

}  // namespace gpu
}  // namespace bc

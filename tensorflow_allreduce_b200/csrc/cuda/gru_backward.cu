// Backward pass of the persistent GRU layer for sm_100a (see gru_persistent.h for the interface).
//
// Work split. Direction d of a layer is run by H/16 blocks (grid.y = direction); block c owns the hidden units [16c, 16c+16) and forms dh of
// these units, step by step backwards. For the recurrent product the blocks work in groups of C that split the reduction length 3H
// among themselves: block q of a group keeps, for ALL 16C units of its group, the weight columns of its range of H/C units (three gates) in
// tensor memory for the whole sequence. Each time step a block
//   1. polls dh of its range in a ring in global memory, multiplies it with the factors of the three gates and puts the products, the
//      gradients of the pre-activations, into shared memory in the 128-byte swizzle,
//   2. multiplies with tcgen05.mma (TF32 operands): the weights are the M side, the batch is the N side, K = 8 per instruction,
//   3. reads the accumulator back (tcgen05.ld: a lane is a weight row, a column a batch entry) and sends every other member of the
//      group the partial sums of that member's units,
//   4. adds up the C partial sums of its own units and puts dh of the next step into the ring.
//
// The factors do not depend on dh: with c = (1 - z)(1 - n^2) they are c hn r (1 - r), (h' - n) z (1 - z), c r (and c and z for the block's
// own outputs). The forward pass writes them (five planes [t][batch][5][H]), and a loader fetches those of the next step
// while it waits. So one value per unit and batch entry has to travel between the blocks instead of three.
//
// What bounds a step (B200): the chain dh published -> seen by the other blocks -> tensor core -> partial sums published -> seen by their owner.
//   * A store by one SM is seen by a relaxed polling load of another after 740 cycles on average, 950 at most; with a release and an
//     acquire on a counter it is 1290 / 1600, and fetching the data behind the counter costs another L2 round trip. So nothing here waits
//     on counters: every word that travels says by itself which step it belongs to.
//       - dh: the lowest of the 24 bits of mantissa is one fixed bit that depends on the step and on whether the unit is even: eight neighbouring words
//         end in 0, 1, 0, 1, ... or 1, 0, 1, 0, ..., the other way round at every second use of their place. Words of another step, and words that were cleared, do
//         not have the pattern. (An infinite dh may arrive as NaN.)
//       - Partial sums need all 32 bits: three of them and the step number share a 16-byte word that is written and read as one
//         access (.b128, single-copy atomic).
//     Both areas have two slots (step parity). Slot reuse is safe without any further exchange: a block writes step s only after partial
//     sums of step s - 1 from its group, which together depend on step s - 1 of EVERY block, and a block produces step s - 1 only after
//     it has consumed all of step s - 2. Stale words of an earlier launch are cleared before the blocks of a direction meet once at the start.
//   * Lines that another SM has just written are slow to read: 128 blocks that read 32 KB each take 1130 cycles when nothing was
//     written, 1406 (the last block 1863) when it was. That is why the volume per block matters, why a loader reads 32 bytes
//     per request, and why nothing is polled before it can be there.
//   * The MMAs are issued as straight-line code: an instruction with operand A in tensor memory takes 16 cycles at N = 32 and 9 at N = 16,
//     whatever M, 12 to issue, but 30 when a loop or a branch stands between it and the one before.
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
constexpr int kGateThreads = 256;     // eight warps: accumulator read-back, exchange, sums, outputs
constexpr int kLoadThreads = 256;     // eight warps: poll the words of dh and form the operand
constexpr int kThreads = kGateThreads + kLoadThreads;
constexpr int kMmaWarp = kGateThreads / 32 - 1;   // the last gate warp, which has no sums to form, issues the MMAs

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
__device__ __forceinline__ void ld_floats8(const float* p, float* v) {
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(p));
}
// dh as it travels: the lowest bit says which step it belongs to.
__device__ __forceinline__ uint32_t tagged(float v, uint32_t tag) { return (__float_as_uint(v) & ~1u) | tag; }
__device__ __forceinline__ bool stale(const Words& v, uint32_t phase) {
  uint32_t d = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) d |= v.w[i] ^ (phase ^ (i & 1));
  return (d & 1u) != 0;
}

// Barrier 1: all gate and loader warps have read the accumulator and sent or stored their part of it; the loaders only arrive. It has no limit, and
// a warp that arrived twice before the others have come once would complete it without them and leave them waiting for good. So gate and
// loader warps come to it once per step whatever waits have run out, and the loaders never before the gate warps have passed it the last
// time: their wait for the block's publication is the one that is never skipped or cut short.
__device__ __forceinline__ void sent_sync() { asm volatile("barrier.cta.sync 1, 512;" ::: "memory"); }
__device__ __forceinline__ void sent_arrive() { asm volatile("barrier.cta.arrive 1, 512;" ::: "memory"); }
__device__ __forceinline__ void gates_sync() { asm volatile("barrier.cta.sync 2, 256;" ::: "memory"); }

__host__ __device__ constexpr int packs_of(int batch) { return (batch + 2) / 3; }   // three partial sums and the step number per 16 bytes

// Where everything of one block lives. C: blocks per group; NB: N of the MMA (16 or 32, at least the batch); H: hidden size.
template <int C, int NB, int H>
struct Plan {
  static constexpr int kRange = H / C;                    // units of one member's K range
  static constexpr int kK = 3 * kRange;                   // [gate][unit]
  static constexpr int kTiles = (kK + kKTile - 1) / kKTile;
  static constexpr int kLaneRows = 4 * C;                 // rows of the group in each quarter of the lanes: row 4C q + i is lane 32q + i
  static constexpr int kParts = kRange >= 64 ? 3 : 1;     // the operand is handed to the tensor core gate by gate, or all at once
  static constexpr int kRangeTiles = (kRange + kKTile - 1) / kKTile;      // the last one may be half
  static constexpr int kLoads = (NB * kRangeTiles * 4 + kLoadThreads - 1) / kLoadThreads;
  static constexpr int kXBytes = kTiles * NB * 128, kOwnBytes = kUnits * packs_of(NB) * 16;
  static constexpr int kSmem = 1024 + kXBytes + kOwnBytes + 256;
  static_assert(NB + kK <= (int)kTmemCols, "the weights live in tensor memory");
};

// Column k0 .. k0 + 15 of member q's K range (k0 a multiple of 16) of row r = 16 owner + unit of the group: W[g * H + unit'][unit]. A run of
// 16 columns stays inside one gate, because a member's range of units is a multiple of 16.
template <int C, int H>
__device__ __forceinline__ void load_weights16(const float* w, int grp, int q, int r, int k0, float* o) {
  constexpr int range = H / C;
  const int g = k0 / range, kk = q * range + k0 - g * range;
  const float* p = w + (size_t)(g * H + kk) * H + grp * C * kUnits + r;
#pragma unroll
  for (int i = 0; i < 16; i++) o[i] = __uint_as_float(to_tf32(__ldg(p + (size_t)i * H)));
}

// RAW: the forward pass has left r, z, n and hn (Params::rsv), and the factors are formed here.
//
// Three kinds of warps, so that no work off the chain of a step (output stores, prefetches) delays the next product: gate warps, loader
// warps, and one warp that issues the MMAs. One barrier each says that a part of the operand is in shared memory (full[part]: loaders ->
// MMA), that the accumulator is complete (done: MMA -> all) and that this block has published (published: gates -> loaders). Nobody
// says that the accumulator has been read: the loaders hand over an operand only after their own part of it and after the publication, which comes
// after the gate warps'.
template <int C, int NB, int H, bool RAW>
__global__ void __launch_bounds__(kThreads, 1) gru_backward_kernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);

  using pl = Plan<C, NB, H>;
  constexpr int kRows = kUnits;            // accumulator rows of a member
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);       // the same for all lanes, and known to be
  const int dir = blockIdx.y, u0 = blockIdx.x * kUnits;
  const int T = p.d.T, B = p.d.B, ND = p.d.ndir;
  const int nblocks = gridDim.x;
  const int grp = blockIdx.x / C, q = blockIdx.x % C;
  const int npacks = packs_of(B);

  uint8_t* x_s = smem;
  uint4* own_s = reinterpret_cast<uint4*>(x_s + pl::kXBytes);                      // this block's own partial sums: [pack][row]
  uint64_t* bar_s = reinterpret_cast<uint64_t*>(x_s + pl::kXBytes + pl::kOwnBytes);  // full[3], done, drain, published
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_s + 6);
  volatile int* abort_s = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t full_bar = smem_u32(bar_s), done_bar = full_bar + 24, drain_bar = full_bar + 32, pub_bar = full_bar + 40;
  const uint32_t x_addr = smem_u32(x_s);

  if (tid == 0) {
    for (int i = 0; i < 3; i++) mbar_init(full_bar + 8 * i, kLoadThreads / 32);
    mbar_init(done_bar, 1);
    mbar_init(drain_bar, 1);
    mbar_init(pub_bar, kGateThreads / 32);
    *abort_s = 0;
    mbar_init_fence();
  }
  if (warp == kMmaWarp) tmem_alloc(tmem_slot, kTmemCols);

  // The part of the ring that this block writes (both slots) and the partial sums that it will receive: cleared, so that nothing of an
  // earlier launch passes for a word of this one. The ring of a direction and slot is [member][tile of 32 units][batch NB][32].
  constexpr uint32_t kMember = pl::kRangeTiles * NB * kKTile, kSlot = kMember * C;
  uint32_t* ring = p.ring + (size_t)dir * 2 * kSlot;
  uint32_t* mine_r = ring + (size_t)(u0 / pl::kRange) * kMember + u0 % pl::kRange / kKTile * (NB * kKTile) + u0 % pl::kRange % kKTile;
  const int xslot = npacks * kRows;                              // 16-byte words of one source and slot
  uint4* xchg = reinterpret_cast<uint4*>(p.ring + (size_t)ND * 2 * kSlot);      // [dir][owner block][source, without the owner][slot 2][pack][row]
  uint4* xin = xchg + ((size_t)dir * nblocks + blockIdx.x) * (C - 1) * 2 * xslot;
  for (int i = tid; i < 2 * kUnits * B; i += kThreads) st_word(mine_r + (i & 1 ? kSlot : 0u) + i / 2 / kUnits * kKTile + i / 2 % kUnits, 0u);
  for (int i = tid; i < (C - 1) * 2 * xslot; i += kThreads) st_pack(xin + i, make_uint4(0, 0, 0, 0));
  for (int i = tid; i < pl::kXBytes / 16; i += kThreads) reinterpret_cast<uint4*>(x_s)[i] = make_uint4(0, 0, 0, 0);
  fence_proxy_async();
  __threadfence();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  Meeting meeting{};
  if (tid == 0) meeting = meet_arrive(p, dir, nblocks);

  // The group's weight rows for this block's K range, rounded to TF32, resident for the whole sequence.
  const int quarter = warp & 3;
  const int lane_row = quarter * pl::kLaneRows + lane;
  const bool row_ok = lane < pl::kLaneRows;
  {
    for (int k0 = 16 * (warp >> 2); k0 < pl::kK; k0 += 64) {
      float v[16];
#pragma unroll
      for (int i = 0; i < 16; i++) v[i] = 0.f;
      if (row_ok) load_weights16<C, H>(p.w_hh[dir], grp, q, lane_row, k0, v);
      __syncwarp();
      tmem_st16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(NB + k0), v);
    }
    tmem_st_wait();
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
  const ptrdiff_t step = dir ? 1 : -1;                  // of time
  const int t_first = dir ? 0 : T - 1, y_row = ND * H;

  // Read-back of the accumulator, by gate and loader warps together: a warp may read the quarter warp % 4 of the lanes, and the four warps of
  // a quarter share the packs of its rows (three batch entries each).
  constexpr int kPacks = packs_of(NB), kPart = (kPacks + 3) / 4;
  const int owner = lane_row / kRows, rr = lane_row % kRows;
  const int pk_lo = (warp >> 2) * kPart, pk_n = max(0, min(kPart, npacks - pk_lo));
  uint4* xout = xchg + (((size_t)dir * nblocks + grp * C + owner) * (C - 1) + (q < owner ? q : q - 1)) * 2 * xslot + pk_lo * kRows + rr;
  auto send = [&](uint32_t tag, uint32_t parity) {
    uint32_t v[3 * kPart];
    tc_fence_after();
    // a few columns past the accumulator's are read as well (they are inside the allocation) and sent as padding
    tc_ld<3 * kPart>(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(3 * pk_lo), v);
    tc_fence_before();
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

  if (ok && warp >= kGateThreads / 32) {
    // ---------------- loaders ----------------
    // Load i of a loader is the 32-byte word lt + 256 i of the member's range: eight units of a batch row. Eight neighbouring lanes write 32 bytes
    // each to two rows of shared memory, to different banks because of the swizzle.
    const int lt = tid - kGateThreads;
    const uint32_t* src0 = ring + (size_t)q * kMember + lt * 8;
    // Load i of a thread is kTilesPerLoad tiles behind load 0; gate g of a range of whole tiles is kRange / 32 tiles behind gate 0.
    constexpr int kTilesPerLoad = kLoadThreads / 4 / NB;
    const int xb = lt / 4 % NB, j0 = lt / 4 / NB * kKTile + lt % 4 * 8;          // batch row, and unit of the range
    uint32_t dst[3];
#pragma unroll
    for (int g = 0; g < 3; g++) {
      const int k = g * pl::kRange + j0;
      dst[g] = x_addr + (uint32_t)((k / kKTile * NB + xb) * 128 + (((k % kKTile / 4) ^ (xb & 7)) << 4));
    }
    bool has[pl::kLoads];
#pragma unroll
    for (int i = 0; i < pl::kLoads; i++) has[i] = xb < B && j0 + i * kTilesPerLoad * kKTile < pl::kRange;
    const int unit = q * pl::kRange + (has[0] ? j0 : 0), fb = has[0] ? xb : 0;
    const size_t frow = (size_t)(dir * T + t_first) * B + fb;
    const float* fac = RAW ? nullptr : p.fac + frow * 5 * H + unit;
    const float4* raw = RAW ? p.rsv + frow * H + unit : nullptr;
    const float* hp = RAW ? p.y + ((ptrdiff_t)t_first + step) * B * y_row + (ptrdiff_t)fb * y_row + dir * H + unit : nullptr;
    float a[pl::kLoads][3][8];
    auto load_factors = [&]() {
#pragma unroll
      for (int i = 0; i < pl::kLoads; i++) {
        if (has[i]) {
          if constexpr (RAW) {
#pragma unroll
            for (int e = 0; e < 8; e++) {
              const Factors f = factors(__ldg(raw + i * kTilesPerLoad * kKTile + e), __ldg(hp + i * kTilesPerLoad * kKTile + e));
              a[i][0][e] = f.r; a[i][1][e] = f.z; a[i][2][e] = f.nr;
            }
          } else {
#pragma unroll
            for (int g = 0; g < 3; g++) ld_floats8(fac + i * kTilesPerLoad * kKTile + g * H, a[i][g]);
          }
        }
      }
      if constexpr (RAW) {
        raw += step * B * H;
        hp += step * B * y_row;
      } else {
        fac += step * B * 5 * H;
      }
    };
    // Cycles from this block's publication to its first poll; see gru_forward.cu. us per step without / with 200 / with 400: H = 1024 B = 32 3.42 /
    // 3.29 / 3.30, B = 8 2.61 / 2.59 / 2.62, B = 1 2.13 / 2.20 / 2.31, H = 128 B = 8 1.73 / 1.86 / 1.97.
    const uint32_t pause = min((uint32_t)(pl::kRange * B * 4) / 40, 300u);
    bool good = true;
    if (T > 1) load_factors();
    // Every step is gone through to the end even when a wait has run out; the waits then end at once, but for the first.
    for (int s = 1; s < T; s++) {
      const uint32_t tag = (uint32_t)s, parity = (uint32_t)(s - 1) & 1, phase = (uint32_t)((s - 1) >> 1) & 1;
      const uint32_t* src = src0 + (parity ? kSlot : 0u);
      // Not before this block has published its own words of the step, and then only when the others' are about to
      // arrive: polling takes L2 bandwidth from the blocks that still exchange partial sums.
      // The gate warps always get there: of their waits before it each runs out once, five limits in all.
      if (!lane_wait(pub_bar, parity, 16 * p.timeout_ns + 1000000000ull, nullptr)) good = give_up(kGruTimeoutBlock);
      for (const uint32_t c0 = clock32(); clock32() - c0 < pause;) {
      }
      Words v[pl::kLoads];
#pragma unroll
      for (int i = 0; i < pl::kLoads; i++)
        if (has[i]) ld_words(src + i * (kLoadThreads * 8), v[i]);
      uint32_t spins = 0;
      unsigned long long t0 = 0;
      for (;;) {
        bool missing = false;
#pragma unroll
        for (int i = 0; i < pl::kLoads; i++)
          if (has[i] && stale(v[i], phase)) {
            missing = true;
            ld_words(src + i * (kLoadThreads * 8), v[i]);
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
      for (int g = 0; g < 3; g++) {
#pragma unroll
        for (int i = 0; i < pl::kLoads; i++)
          if (has[i]) {
            Words o;
#pragma unroll
            for (int e = 0; e < 8; e++) o.w[e] = __float_as_uint(__uint_as_float(v[i].w[e]) * a[i][g][e]);
            st_shared2(dst[g] + i * (kTilesPerLoad * NB * 128), o);
          }
        if (g == 2 || pl::kParts == 3) {
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) mbar_arrive(full_bar + 8 * (pl::kParts == 3 ? g : 0));
        }
      }
      // The MMAs have read the operand area and written the accumulator.
      if (good && !lane_wait(done_bar, parity, 4 * p.timeout_ns, abort_s)) good = *abort_s ? false : give_up(kGruTimeoutMma);
      if (__all_sync(0xffffffffu, good)) send(tag, parity);
      else good = false;
      sent_arrive();
      if (s + 1 < T) load_factors();            // behind the partial sums, which somebody waits for
    }
  } else if (ok) {
    // ---------------- gates ----------------
    // Thread (u, pk) handles unit u0 + u for the batch entries b0 .. b0 + mine - 1.
    const int u = tid & 15, pk = tid >> 4, b0 = 3 * pk;
    const int mine = pk < npacks ? min(3, B - b0) : 0;
    const uint4* xmine = xin + pk * kRows + u;
    const uint4* own_mine = own_s + pk * kRows + u;
    const bool stamping = p.prof && tid == 0 && blockIdx.x == 0 && blockIdx.y == 0;
    auto stamp = [&](int s, int i) {
      if (stamping) p.prof[(size_t)s * 8 + i] = gtimer();
    };

    // Recurrent product number s: wait for the MMAs, exchange inside the group; acc[j] receives the sum for batch entry b0 + j.
    // `good` falls when one of this thread's waits has run out; the steps are gone through to the end all the same.
    bool good = true;
    const uint64_t b_desc = operand_desc(x_addr);
    bool mma_ok = true;       // the same for all lanes
    auto product = [&](int s, float* acc) {
      const uint32_t tag = (uint32_t)s + 1, parity = (uint32_t)s & 1;
      if (warp == kMmaWarp) {
#pragma unroll
        for (int g = 0; g < pl::kParts; g++) {
          mma_ok = mma_ok && bar_wait(full_bar + 8 * g, parity, 4 * p.timeout_ns, abort_s);
          if (!mma_ok) break;
          if (g == 0) tc_fence_after();
          if (elect_one()) {
            constexpr uint32_t kIdesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(NB >> 3) << 17) | (8u << 24);     // M = 128
            constexpr int kSteps = pl::kK / 8 / pl::kParts;
#pragma unroll
            for (int i = 0; i < kSteps; i++) {
              const int k = 8 * (g * kSteps + i);
              tc_mma_ts(tmem, tmem + NB + k, b_desc + (uint64_t)(k / kKTile * (NB * 8) + k % kKTile / 4), kIdesc, k > 0);
            }
          }
          __syncwarp();
        }
        if (mma_ok && elect_one()) tc_commit(done_bar);
        if (!mma_ok && lane == 0 && !*abort_s) give_up(kGruTimeoutBlock);
        __syncwarp();
      }
      if (good && !lane_wait(done_bar, parity, 4 * p.timeout_ns, abort_s)) good = *abort_s ? false : give_up(kGruTimeoutMma);
      stamp(s, 1);
      if (__all_sync(0xffffffffu, good)) send(tag, parity);
      else good = false;
      sent_sync();
      stamp(s, 2);
      uint4 v[C - 1];
      if (mine > 0) {
        const uint4* in = xmine + (parity ? xslot : 0);
#pragma unroll
        for (int i = 0; i < C - 1; i++) v[i] = ld_pack(in + i * 2 * xslot);
        uint32_t spins = 0;
        unsigned long long t0 = 0;
        for (;;) {
          bool missing = false;
#pragma unroll
          for (int i = 0; i < C - 1; i++)
            if (v[i].w != tag) {
              missing = true;
              v[i] = ld_pack(in + i * 2 * xslot);
            }
          if (!missing || !good) break;
          if (((++spins) & 63) == 0) {
            const unsigned long long now = gtimer();
            if (t0 == 0) t0 = now;
            if (*abort_s) good = false;
            else if (now - t0 > p.timeout_ns) good = give_up(kGruTimeoutGrid);
          }
        }
      }
      if (mine > 0) {
        const uint4 o = own_mine[0];
        acc[0] = __uint_as_float(o.x);
        acc[1] = __uint_as_float(o.y);
        acc[2] = __uint_as_float(o.z);
#pragma unroll
        for (int i = 0; i < C - 1; i++) {
          acc[0] += __uint_as_float(v[i].x);
          acc[1] += __uint_as_float(v[i].y);
          acc[2] += __uint_as_float(v[i].z);
        }
      }
      stamp(s, 3);
    };

    const int dg_row = ND * 4 * H, bb = mine > 0 ? b0 : 0;
    const size_t row = (size_t)(dir * T + t_first) * B + bb;
    const float* fac_p = RAW ? nullptr : p.fac + row * 5 * H + u0 + u;
    const float4* rsv_p = RAW ? p.rsv + row * H + u0 + u : nullptr;
    const float* hp_p = RAW ? p.y + ((ptrdiff_t)t_first + step) * B * y_row + (ptrdiff_t)bb * y_row + dir * H + u0 + u : nullptr;   // h of the step before in the forward pass
    const float* dy_p = p.dy + ((size_t)t_first * B + bb) * y_row + dir * H + u0 + u;
    float* dg_p = p.dg + ((size_t)t_first * B + bb) * dg_row + dir * 3 * H + u0 + u;
    const int dnr_off = (ND * 3 - dir * 2) * H;       // from (dir * 3) * H to (ND * 3 + dir) * H
    uint32_t* ring_p = mine_r + bb * kKTile + u;
    Factors f[3] = {};
    float dy[3] = {0.f, 0.f, 0.f};
    auto load_inputs = [&](bool has_prev) {
#pragma unroll
      for (int j = 0; j < 3; j++)
        if (j < mine) {
          if constexpr (RAW) {
            f[j] = factors(__ldg(rsv_p + j * H), has_prev ? __ldg(hp_p + j * y_row) : 0.f);
          } else {
            const float* o = fac_p + j * 5 * H;
            f[j].r = __ldg(o); f[j].z = __ldg(o + H); f[j].nr = __ldg(o + 2 * H); f[j].n = __ldg(o + 3 * H); f[j].keep = __ldg(o + 4 * H);
          }
          dy[j] = __ldg(dy_p + j * y_row);
        }
      if constexpr (RAW) {
        rsv_p += step * B * H;
        hp_p += step * B * y_row;
      } else {
        fac_p += step * B * 5 * H;
      }
      dy_p += step * B * y_row;
    };
    float carry[3] = {0.f, 0.f, 0.f};                                      // recurrent part of dh
    float sum[4] = {0.f, 0.f, 0.f, 0.f}, part[4] = {0.f, 0.f, 0.f, 0.f};   // bias gradients, in runs of 16 steps
    load_inputs(T > 1);
    for (int s = 0; s < T; s++) {
      stamp(s, 0);
      float dh[3];
#pragma unroll
      for (int j = 0; j < 3; j++) dh[j] = dy[j] + carry[j];
      if (s + 1 < T) {
        uint32_t* o = ring_p + ((s & 1) ? kSlot : 0u);
        const uint32_t tag = ((uint32_t)(s >> 1) ^ (uint32_t)u) & 1u;
#pragma unroll
        for (int j = 0; j < 3; j++)
          if (j < mine) st_word(o + j * kKTile, tagged(dh[j], tag));
        // This block's words of a step are on their way: its loaders may begin to poll the others'.
        __syncwarp();
        if (lane == 0) mbar_arrive(pub_bar);
      }
      stamp(s, 4);
      // The peers do not wait for what follows.
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const float g[4] = {dh[j] * f[j].r, dh[j] * f[j].z, dh[j] * f[j].n, dh[j] * f[j].nr};
        carry[j] = dh[j] * f[j].keep;
        if (j < mine) {
          float* o = dg_p + j * dg_row;
#pragma unroll
          for (int k = 0; k < 3; k++) o[k * H] = g[k];
          o[dnr_off] = g[3];
#pragma unroll
          for (int k = 0; k < 4; k++) part[k] += g[k];
        }
      }
      dg_p += step * B * dg_row;
      if ((s & 15) == 15) {
#pragma unroll
        for (int k = 0; k < 4; k++) { sum[k] += part[k]; part[k] = 0.f; }
      }
      if (s + 1 < T) {
        load_inputs(s + 2 < T);
        float acc[3] = {};
        product(s, acc);
#pragma unroll
        for (int j = 0; j < 3; j++) carry[j] += acc[j];
      }
    }
    if (warp == kMmaWarp) {
      if (elect_one()) {
        // Nothing may be in flight when tensor memory is freed, whatever this or another warp has not waited for.
        tc_commit(drain_bar);
        mbar_drain(drain_bar, 0);
      }
      __syncwarp();
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
  if (warp == kMmaWarp) tmem_free(tmem, kTmemCols);
}

template <int C, int NB, int H, bool RAW>
cudaError_t launch_with(const Params& p, cudaStream_t stream) {
  auto kernel = gru_backward_kernel<C, NB, H, RAW>;
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
  return cudaLaunchCooperativeKernel((const void*)kernel, dim3(H / kUnits, p.d.ndir), dim3(kThreads), args,
                                     (size_t)std::max(Plan<C, NB, H>::kSmem, kMinSmem), stream);
}

template <int C, int NB, int H>
cudaError_t launch_as(const Params& p, cudaStream_t stream) {
  return p.fac ? launch_with<C, NB, H, false>(p, stream) : launch_with<C, NB, H, true>(p, stream);
}

// Blocks per group: eight, the 128 rows of an MMA. us per step with groups of 8 / 4 (/ 2): B = 32 H = 512 2.91 / 2.99, 384 2.72 / 2.82, 256 2.50 /
// 2.63 / 2.61, 128 2.12 / 2.12 / 2.11; B = 8 H = 512 2.46 / 2.41, 256 2.07 / 2.17 / 2.04, 128 1.73 / 1.89 / 1.84. Groups of four where the
// exchange memory does not hold the partial sums of eight. (With less than eight and H = 640 or more the weights do not fit.)
template <int NB, int H>
cudaError_t launch(const Params& p, cudaStream_t stream) {
  return launch_as<NB == 32 && H <= 256 ? 4 : 8, NB, H>(p, stream);
}

}  // namespace

namespace gru {

cudaError_t launch_backward(const Params& p, cudaStream_t stream) {
  auto with = [&](auto h) { return p.d.B <= 16 ? launch<16, decltype(h)::value>(p, stream) : launch<32, decltype(h)::value>(p, stream); };
  switch (p.d.H) {
    case 128: return with(std::integral_constant<int, 128>{});
    case 256: return with(std::integral_constant<int, 256>{});
    case 384: return with(std::integral_constant<int, 384>{});
    case 512: return with(std::integral_constant<int, 512>{});
    case 640: return with(std::integral_constant<int, 640>{});
    case 768: return with(std::integral_constant<int, 768>{});
    case 896: return with(std::integral_constant<int, 896>{});
    case 1024: return with(std::integral_constant<int, 1024>{});
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace gru
}  // namespace gpu
}  // namespace bc

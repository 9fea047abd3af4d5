// Operators G, S and D for 16-bit tensors as one persistent, warp-specialised kernel (sm_100a), on one CTA or a pair of CTAs per tile.
//
//   warps 0..7    gather producers: index-driven row copies into the stage ring, 16-byte cp.async on a CTA of its own, four rows by
//                 TMA (tile::gather4) in a pair; in a scatter whose slot rows come as boxes they have nothing to gather and join the
//                 read-out
//   warps 8..15   read-out: tensor memory -> stores (G, D) / red.global.add (S)
//   warp  16      tensor-memory allocation; four tcgen05.mma per stage, issued by the leader of a pair for both (cta_group::2)
//   warp  17      the TMA box loads of everything that is not gathered; announces the bytes of a stage
//   warps 18, 19  look up the rows of the tiles to come: G, S source rows (18) and destination rows (19); D the contraction rows
//
// A unit of work is one accumulator tile of 128 x BN per CTA (256 x BN per pair); CTAs (one per SM) walk the units, the stage ring
// runs on across them and the accumulator is double-buffered in tensor memory, so neither set-up nor read-out stands between two tiles.
//   G  rows = expert rows, token rows through Ind (gathered);     columns = W[e] (boxes)
//   S  rows = expert rows, slot rows (boxes where 128 rows are whole batch elements or parts of one, else gathered);  columns = W[e]
//   D  contraction = expert rows; one operand the gathered token rows, the other the slot rows (boxes under the same condition for
//      64 rows, else gathered).  Either may be the one whose features are the accumulator's rows.
//
// Everything a pair stages comes through the TMA units, and both CTAs' bytes are counted by the leader's barrier
// (cp.async.bulk.tensor with cta_group::2): the leader's MMAs read the peer's shared memory behind nothing but that count.  Rows
// copied there by cp.async would have to be handed over by a thread of the peer, with a proxy fence and an arrival that releases at
// cluster scope: 1400 clocks a stage (B=512 as below: 10.4 ms a pass against 8.0; with three threads handing over in turn 8.5).
// Accumulators go back to the leader by relaxed arrivals: nothing written is handed over, and tcgen05.wait::ld has returned, so
// the loads have their values before the arrival is made.
//
// What bounds the main loop is shared-memory bandwidth and the tensor core together: a stage (64 contraction elements) of a 128 x 256
// tile is 48 KB written and 48 KB read by its four MMAs, 750 clocks at 128 bytes per clock against 512 clocks of tensor work; a pair
// stages half the columns per CTA and moves 64 KB, 512 clocks.  16-byte cp.async costs the load/store unit about 10 clocks per warp
// instruction (320 a stage of G), side by side with the TMA unit; a pair's gathers take the TMA units about as long.  Everything else has to stay out of the way: a satisfied barrier
// wait takes 150 clocks and every dependent instruction of a lone warp 5-10, so nothing on a per-stage or per-tile path divides, the
// issuing warps run converged (see mbar_wait_all) and ids are looked up elsewhere.
// T=1024, E=64, K=64, I=1024, J=256, bf16: B=64 G and dY (weights [E, N, C]) 105-110 us, D 119-123 (138 before its gathers came in groups, segment by
// segment); B=512, under the power cap, G and dY 850-950 us = 1.15-1.3 PFLOP/s, D 1050-1150.  S as whole calls: B=64 174 us, B=512 1340, 150 of which
// fill the output (its rows loaded for every column tile instead of kept: 194 and 1450 before that fill took 30 us less).
#include <algorithm>
#include <type_traits>

#include "egs_tcgen05.cuh"

namespace egs {

namespace {

constexpr int kProdWarps = 8, kProdThreads = kProdWarps * 32;
constexpr int kEpiWarps = 8;
constexpr int kMmaWarp = kProdWarps + kEpiWarps, kTmaWarp = kMmaWarp + 1;
constexpr int kIndexWarp = kTmaWarp + 1, kIndexWarps = 2;
constexpr int kDenseThreads = (kIndexWarp + kIndexWarps) * 32;
constexpr int kStep = 64;                          // contraction elements per stage
constexpr uint32_t kDenseHeader = 1024;
constexpr int kBatch = 256;                        // D: contraction rows whose ids are looked up at a time (four steps)
// D: two batches of token rows; without TMA boxes for the slot rows two of those as well.  (Sized so that four stages of a
// 128 x 256 tile still fit beside it with TMA boxes: three stages cost a quarter of the rate.)
__host__ __device__ constexpr uint32_t table_bytes(bool slots) { return (slots ? 4u : 2u) * kBatch * 4u; }
// G, S: source rows of two units, then destination rows of two units (-1: none)
constexpr uint32_t kRowTable = 4u * kTileM * 4u;
constexpr uint32_t kMTile = 16384;                 // bytes of the 128-wide operand: 128 rows x 64 elements, or 64 rows x 128
constexpr uint32_t kSeg = kStep * 128u;            // one 64-column segment of a 64-row tile
__host__ __device__ constexpr uint32_t epi_bytes(bool wide) { return (wide ? kProdWarps + kEpiWarps : kEpiWarps) * 4096u; }       // transposes of the read-out
constexpr size_t kSmemMax = 227 * 1024;
constexpr int kSms = 148;

enum { kOpGather = 0, kOpScatter = 1, kOpDweight = 2 };

struct __align__(16) DenseHeader {
  unsigned long long full[kMaxStages];
  unsigned long long empty[kMaxStages];
  unsigned long long acc_full[2];
  unsigned long long acc_empty[2];
  unsigned long long ids_full[2];
  unsigned long long ids_empty[2];
  unsigned long long dst_full[2];
  unsigned long long dst_empty[2];
  unsigned long long drain;
  unsigned long long last;               // ... and the column tiles that this CTA was the last to add to
  uint32_t tmem_base;
  uint32_t abort_flag;
  uint32_t reached;                      // S whose rows stay: step that the TMA warp has come to, of those that begin a row block or follow the last
  int rounds;                            // S: float32 rows are to be rounded here ...
};
static_assert(sizeof(DenseHeader) <= kDenseHeader, "header does not fit");

struct DenseParams {
  const void* Rows;   // G, D: token rows; S: slot rows
  const void* Slot;   // D: slot rows
  const void* bias;   // G, S: [E, N] or NULL
  const void* Ind;
  void* Out;          // G: slot rows; S: token rows; D: the gradient
  float* acc;         // S: float32 rows; D: float32 sums when splits > 1
  int* plan;          // S: PlanWords
  int rounds;         // S: the kernel rounds float32 rows itself
  StatusRef status;
  int B, T, E, K, M;
  int C, N;           // G, S: contraction and produced width; D: features of the operand along the accumulator's rows / columns
  int nc;             // G, S: 1 = weights [E, N, C]
  int index_dtype;
  int BN, stages;
  int tiles_m, tiles_n, units;           // row blocks, column tiles
  int full_waves;                        // S: units of all column tiles of a row block that every CTA (pair) has, before the others
  int group, groups_n;                   // column tiles of one of the other units, units of a row block
  int a_slots;                           // tiles of the 128-wide operand that are kept: `stages`, or a scatter's whole row block
  int readers;                           // read-out warps
  Div r1, r2;                            // radices of the unit number, see Walk
  Div stride;                            // CTAs or pairs
  Div by_k, by_group, by_tiles;          // K, groups_n, tiles_n
  int step_full[3], step[4];             // digits of the stride: whole row blocks, other units
  int splits, rows_per_split;            // D
  int swap;           // D: 1 = the slot rows' features are the accumulator's rows
  int lane_rows;      // D: 1 = the output's rows are the accumulator's rows
  int tma_rows;       // S, D: slot rows come by TMA
  int whole, boxes;   // weights [E, C, N], D's slot rows: boxes of all 64-column segments of a tile (see whole_segments), boxes of a tile
  int half;           // columns of a tile one CTA stages: BN, or BN / 2 in a pair
  int after_own;      // see launch_kernel
  int tail, tail_bn;                     // G on pairs: units of half a tile in the last wave (0: none), width of the first half (see plan_tail)
};

// Position in the stage ring.
struct Cursor {
  int slot = 0, round = 0;
  __device__ __forceinline__ void next(int stages) {
    if (++slot == stages) {
      slot = 0;
      ++round;
    }
  }
};

// The tiles of a CTA or pair.  A unit is a number in a mixed radix - column tile; row block of a group, expert, group (G, S) or row block,
// row range, expert (D) - units go out `stride` apart and are advanced by adding the stride's digits: three divisions a unit (1000
// clocks and more) in the lanes that feed the tensor core were a fifth of the time of a tile with eight steps.
// The last wave of G on pairs may be units of half a tile (see plan_tail).
// A scatter whose rows may stay has units of several column tiles: all of a row block's for as many whole waves as there are, and
// groups of them, so that the last wave is even, for the row blocks that are left.
template <int OP, bool PAIR, bool KEEP>
struct Walk {
  int left;                    // units to come, this one included
  int m0, n0, e, split;        // this CTA's 128 rows, the first column of the tile, expert, row range
  int j, tiles, tile;          // tiles of the unit before this one, its tiles, this one's place among them
  int full, d0, d1, d2, d3;
  int bn;                      // width of the unit's tile
  const DenseParams& p;
  static constexpr bool kTails = PAIR && OP == kOpGather;
  __device__ __forceinline__ explicit Walk(const DenseParams& q) : p(q) {
    const int c = PAIR ? blockIdx.x >> 1 : blockIdx.x, s = p.stride.d;
    bn = p.BN;
    full = KEEP || (kTails && p.tail > 0) ? p.full_waves : 0;
    const int rest = p.units - full * s * p.groups_n;    // (p.units counts the units as if all were of the second kind)
    left = kTails && full > 0 ? full + (c < p.tail ? 1 : 0) : full + (c < rest ? p.stride.quotient(rest - c + s - 1) : 0);
    begin(0);
  }
  // the first unit of the row blocks from `block` on
  __device__ __forceinline__ void begin(int block) {
    int u = PAIR ? blockIdx.x >> 1 : blockIdx.x;
    if (!KEEP) u += block;               // (of which each has one unit here)
    d0 = KEEP && full > 0 ? 0 : p.by_group.remainder(u);
    if (KEEP) u += block;
    d1 = p.r1.remainder(u);
    d2 = p.r2.remainder(u);
    d3 = u;
    place();
  }
  __device__ __forceinline__ void place() {
    const int mt = OP == kOpDweight ? d1 : d3 * p.r1.d + d1;
    e = OP == kOpDweight ? d3 : d2;
    split = OP == kOpDweight ? d2 : 0;
    m0 = PAIR ? mt * 2 * kTileM + static_cast<int>(blockIdx.x & 1) * kTileM : mt * kTileM;
    if (!KEEP) {
      n0 = d0 * p.BN;
      return;
    }
    // A scatter's units begin at different column tiles: CTAs in flight have experts of the same token rows, and additions that
    // meet in one part of them hold each other up.
    const int group = full > 0 ? p.tiles_n : p.group;
    int turn = e;
    j = 0;
    tiles = min(group, p.tiles_n - d0 * group);
    tile = p.by_tiles.remainder(turn);
    if (tile >= tiles) tile = 0;
    n0 = (d0 * group + tile) * p.BN;
  }
  __device__ __forceinline__ void next() {
    if (KEEP && ++j < tiles) {
      const bool wrap = ++tile == tiles;
      n0 += wrap ? (1 - tiles) * p.BN : p.BN;
      if (wrap) tile = 0;
      return;
    }
    --left;
    if (kTails && full > 0 && --full == 0) {
      const int c = blockIdx.x >> 1, second = c & 1;
      begin(p.full_waves * p.stride.d + (c >> 1) - c);
      n0 += second * p.tail_bn;
      bn = second ? p.BN - p.tail_bn : p.tail_bn;
      return;
    }
    const bool whole = KEEP && full > 0;
    if (whole && --full == 0) {
      begin(p.full_waves * p.stride.d);
      return;
    }
    d0 += whole ? 0 : p.step[0];
    d1 += whole ? p.step_full[0] : p.step[1];
    d2 += whole ? p.step_full[1] : p.step[2];
    d3 += whole ? p.step_full[2] : p.step[3];
    if (!whole && d0 >= p.groups_n) { d0 -= p.groups_n; ++d1; }
    if (d1 >= p.r1.d) { d1 -= p.r1.d; ++d2; }
    if (d2 >= p.r2.d) { d2 -= p.r2.d; ++d3; }
    place();
  }
  __device__ __forceinline__ int steps() const {
    if (OP != kOpDweight) return (p.C + kStep - 1) / kStep;
    return (min(p.rows_per_split, p.M - split * p.rows_per_split) + kStep - 1) / kStep;
  }
  // width of the tile's MMA (the last tile of a row may be narrower), and the first column this CTA stages
  __device__ __forceinline__ int width() const {
    const int rest = p.N - n0;
    return min(kTails ? bn : p.BN, PAIR ? (rest + 31) & ~31 : (rest + 15) & ~15);
  }
  // 64-column segments of the tile that a CTA stages
  __device__ __forceinline__ int segs() const { return ((PAIR ? bn >> 1 : bn) + 63) >> 6; }
  __device__ __forceinline__ int first_column() const { return PAIR && (blockIdx.x & 1) ? n0 + width() / 2 : n0; }
};

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const void* map, int x, int y, int z, int w, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
      : "memory");
}

// Rounds the float32 rows of a small scatter that sums in those, behind the barrier of the common exit.  A column tile is rounded by the CTA that
// is the last to have added to it: one CTA for all of them took 1.5 us more at 16 Ki elements and 3.5 at 64 Ki.  Nobody waits for another CTA,
// which may have yet to find room beside another stream's kernels.
template <typename T, bool PAIR>
__device__ __noinline__ void round_rows(const DenseParams& p, DenseHeader* hdr) {
  const int tid = threadIdx.x;
  if (tid < p.tiles_n) {
    int added = 0;                                   // units of column tile `tid` that this CTA has had
    for (int u = PAIR ? blockIdx.x >> 1 : blockIdx.x; u < p.units; u += p.stride.d) added += u % p.tiles_n == tid;
    __threadfence();
    const int all = p.units / p.tiles_n * (PAIR ? 2 : 1);
    if (added > 0 && atomicAdd(p.plan + kPlanAdded + tid, added) + added == all) atomicOr(&hdr->last, 1ull << tid);
    __threadfence();
  }
  __syncthreads();
  T* out = static_cast<T*>(p.Out);
  for (unsigned long long tiles = hdr->last; tiles != 0; tiles &= tiles - 1) {
    const int n0 = (__ffsll(static_cast<long long>(tiles)) - 1) * p.BN, chunks = min(p.BN, p.N - n0) / 8;      // of eight columns a row
    const int n = p.B * p.T * chunks;                // (see kRoundInKernel)
    constexpr int kAtOnce = 4;
    for (int i0 = tid; i0 < n; i0 += kAtOnce * kDenseThreads) {
      int at[kAtOnce];
      float4 v[2 * kAtOnce];
#pragma unroll
      for (int j = 0; j < kAtOnce; ++j) {
        const int i = i0 + j * kDenseThreads, row = i / chunks;
        at[j] = i < n ? row * p.N + n0 + (i - row * chunks) * 8 : -1;
        if (at[j] >= 0) {
          v[2 * j] = __ldcg(reinterpret_cast<const float4*>(p.acc + at[j]));
          v[2 * j + 1] = __ldcg(reinterpret_cast<const float4*>(p.acc + at[j]) + 1);
        }
      }
#pragma unroll
      for (int j = 0; j < kAtOnce; ++j) {
        const float4 a = v[2 * j], b = v[2 * j + 1];
        if (at[j] >= 0)
          *reinterpret_cast<uint4*>(out + at[j]) =
              make_uint4(pack2(out, __float_as_uint(a.x), __float_as_uint(a.y)), pack2(out, __float_as_uint(a.z), __float_as_uint(a.w)),
                         pack2(out, __float_as_uint(b.x), __float_as_uint(b.y)), pack2(out, __float_as_uint(b.z), __float_as_uint(b.w)));
      }
    }
  }
}

// (PAIR: counted by the leader's barrier, see tma_load_3d_pair)
template <bool PAIR>
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const void* map, int x, int y, int z, int v, int w, uint32_t bar) {
  if (PAIR)
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(v), "r"(w), "r"(bar)
        : "memory");
  else
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(v), "r"(w), "r"(bar)
        : "memory");
}

// KEEP: a scatter whose rows stay for several column tiles (see pick_tile).  An instance of its own: with the slots of kept rows and the
// walk over both kinds of units in the lanes that issue loads and MMAs, scatters that keep nothing took 3-7 % longer (bf16, 64 experts
// of 5760 rows, 128 -> 520 features: 181 us without, 193 with).
template <typename T, int OP, bool PAIR, bool KEEP>
__global__ void __cluster_dims__(PAIR ? 2 : 1, 1, 1) __launch_bounds__(kDenseThreads, 1) dense16_kernel(const __grid_constant__ DenseParams p, const __grid_constant__ TensorMap3 map_w,
                                                                   const __grid_constant__ TensorMap3 map_rows) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  DenseHeader* hdr = reinterpret_cast<DenseHeader*>(smem_raw);
  const uint32_t smem0 = smem_u32(smem_raw);
  const uint32_t epi0 = smem0 + kDenseHeader + (OP == kOpDweight ? table_bytes(!p.tma_rows) : kRowTable);
  const bool gathers = OP != kOpScatter || !p.tma_rows;
  const bool has_cp = !PAIR && gathers;
  const int readers = p.readers;                                        // read-out warps: producers with nothing to gather may join
  const uint32_t ring0 = epi0 + epi_bytes(readers > kEpiWarps);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool leader = !PAIR || (blockIdx.x & 1) == 0;
  // (in a pair the leader's also announces what the producers gather; a warp without a part in a stage must not follow the ring, see is_mine)
  const bool has_tma = OP != kOpDweight || p.tma_rows || (PAIR && leader);
  const int nseg = (p.half + 63) >> 6;
  const uint32_t n_bytes = (OP != kOpDweight && p.nc) ? static_cast<uint32_t>(p.half) * 128u : static_cast<uint32_t>(nseg) * kSeg;
  const uint32_t stage_bytes = kMTile + n_bytes;
  const int stages = p.stages;
  // a kept tile of the 128-wide operand: with the stages, those beyond their number behind them
  auto a_tile = [&](int slot) {
    return ring0 + (!KEEP || slot < stages ? static_cast<uint32_t>(slot) * stage_bytes : static_cast<uint32_t>(stages) * stage_bytes + static_cast<uint32_t>(slot - stages) * kMTile);
  };
  const uint32_t acc_cols = tmem_cols_for(p.BN);
  const uint32_t tmem_cols = 2u * acc_cols;
  volatile uint32_t* abort_flag = &hdr->abort_flag;

  if (tid == 0) {
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(smem_u32(&hdr->full[s]), (has_cp ? kProdThreads : 0) + (PAIR || has_tma ? 1 : 0));      // (a pair's: the leader's copy is used)
      mbar_init(smem_u32(&hdr->empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&hdr->acc_full[b]), 1);
      mbar_init(smem_u32(&hdr->acc_empty[b]), PAIR ? 2 * readers : readers);       // (a pair's: the leader's copy is used)
      mbar_init(smem_u32(&hdr->ids_full[b]), OP == kOpDweight ? kIndexWarps * 32 : 32);
      mbar_init(smem_u32(&hdr->dst_full[b]), 32);
      mbar_init(smem_u32(&hdr->dst_empty[b]), readers);
      mbar_init(smem_u32(&hdr->ids_empty[b]), kProdWarps);
    }
    mbar_init(smem_u32(&hdr->drain), 1);
    fence_mbar_init();
    if (!p.after_own) pdl_wait();
    hdr->abort_flag = p.status.timed_out() ? 1u : 0u;
    hdr->rounds = 0;
    hdr->last = 0ull;
    hdr->reached = 0u;
    if (smem_misaligned(smem_raw)) {
      hdr->abort_flag = 1u;
      p.status.report(EGS_STATUS_INTERNAL);
    }
  }
  if (PAIR) __syncthreads();
  if (warp == kMmaWarp) {
    if (PAIR) {
      tmem_alloc2(smem_u32(&hdr->tmem_base), tmem_cols);
      tmem_relinquish2();
    } else {
      tmem_alloc(smem_u32(&hdr->tmem_base), tmem_cols);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();          // both CTAs' barriers are initialised before anything crosses the pair
  tc_fence_after();
  const uint32_t tmem_base = hdr->tmem_base;
  if (!p.after_own) pdl_wait();

  if (hdr->abort_flag != 0u) {
    pdl_wait();                          // (and fall through to the common exit)
  } else if (PAIR && warp < kProdWarps && gathers) {
    // =========================== gather producers of a pair ===========================
    // Rows come four at a time (tile::gather4).  In D two groups of four warps share the stages, a warp has a quarter of a stage's
    // rows, and loads them segment by segment: a warp's loads one after the other go to one stretch of shared memory, and what a step
    // costs a warp beside them - ids, the barrier, coordinates moved to uniform registers - it has two steps' time for.  With eight
    // rows of both segments in turn for every stage, the gathers alone of a step took 860 clocks (with everything else 974, now 800), more
    // than its MMAs: bf16, 64 experts of 1024 rows, 2048 x 512 features 132 us; eight rows segment by segment 120; in two groups 116.
    // G and S, whose warps keep their rows for a whole tile, gain nothing from groups.
    constexpr int kGroups = OP == kOpDweight ? 2 : 1, kParts = kProdWarps / kGroups;
    const int group = warp & (kGroups - 1), part = warp / kGroups;
    const uint32_t table = smem0 + kDenseHeader;
    auto get4 = [](uint32_t a, int (&r)[4]) {
      asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
    };
    Cursor at;
    bool alive = true;
    auto wait_free = [&]() {             // for the stage at `at`; its barrier (the leader's) and its first byte here; moves on
      if (at.round > 0) alive = mbar_wait_all(smem_u32(&hdr->empty[at.slot]), (at.round - 1) & 1, abort_flag, p.status.word);
    };
    // Whether the stage at `at` is this warp's.  A group has every other slot of the ring, not every other step: with an odd number of stages
    // the groups would meet each barrier in turn, and a warp that is late to look at a phase whose stage another group loads finds the one
    // after it done as well, which a parity cannot tell from neither being done.
    auto is_mine = [&]() { return kGroups == 1 || (at.slot & (kGroups - 1)) == group; };
    // Rows that stay are loaded with their first column tile only.  With the others these warps have no part in the stages, and one that is late by
    // a turn of the ring finds the phase after the one that it looks for done as well, which a parity cannot tell from neither being done.  It would
    // wait forever, but the TMA warp, which has a part in every stage, says when it has come to the next row block: all phases before are done then.
    auto wait_passed = [&](uint32_t next_block) {          // for the stage at `at`, or that the step of this number has been reached
      if (at.round == 0) return;
      const uint32_t bar = smem_u32(&hdr->empty[at.slot]), parity = (at.round - 1) & 1;
      const long long t0 = clock64();
      while (!__all_sync(0xffffffffu, mbar_try(bar, parity) != 0u)) {
        uint32_t reached;
        asm volatile("ld.acquire.cta.shared::cta.b32 %0, [%1];" : "=r"(reached) : "r"(smem_u32(&hdr->reached)) : "memory");
        if (__all_sync(0xffffffffu, reached >= next_block)) return;
        if (!__any_sync(0xffffffffu, *abort_flag != 0u || clock64() - t0 > kWaitLimitCycles)) continue;
        if (lane == 0 && !*abort_flag) {
          *abort_flag = 1u;
          p.status.report(EGS_STATUS_PIPELINE_TIMEOUT);
        }
        alive = false;
        return;
      }
    };
    const uint32_t full0 = map_to_cta(smem_u32(&hdr->full[0]), 0);
    if constexpr (OP != kOpDweight) {
      constexpr int kQuads = kTileM / kParts / 4;        // G, S: 16 rows a warp
      const int steps = (p.C + kStep - 1) / kStep;
      int t = 0, a_slot = 0;
      uint32_t done = 0;                                 // steps up to the end of this tile
      for (Walk<OP, PAIR, KEEP> u(p); u.left > 0 && alive; u.next(), ++t) {
        alive = mbar_wait_all(smem_u32(&hdr->ids_full[t & 1]), (t >> 1) & 1, abort_flag, p.status.word);
        if (!alive) break;
        int row[kQuads][4];
#pragma unroll
        for (int q = 0; q < kQuads; ++q) get4(table + static_cast<uint32_t>((t & 1) * kTileM + (part * kQuads + q) * 4) * 4u, row[q]);
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&hdr->ids_empty[t & 1]));
        if (KEEP) done += steps;
        for (int k = 0; k < steps; ++k) {
          const bool mine = is_mine();
          if (KEEP && u.j > 0) wait_passed(done + (u.tiles - u.j - 1) * steps);
          else if (mine) wait_free();
          if (!alive) break;
          const int slot = at.slot;
          const uint32_t bar = full0 + slot * 8u;
          at.next(stages);
          if (KEEP && u.j > 0) continue;     // (the rows are there)
          const uint32_t dst = a_tile(KEEP ? a_slot : slot) + static_cast<uint32_t>(part * kQuads) * 512u;
          if (KEEP && ++a_slot == p.a_slots) a_slot = 0;
          if (mine && elect_one()) {
#pragma unroll
            for (int q = 0; q < kQuads; ++q) tma_gather4_pair(dst + q * 512u, &map_rows, k * kStep, row[q][0], row[q][1], row[q][2], row[q][3], bar);
          }
        }
      }
    } else {
      constexpr int kQuads = kStep / kParts / 4;         // 16 rows a warp
      const uint32_t g_dst = p.swap ? kMTile : 0u, s_dst = p.swap ? 0u : kMTile;
      const int g_seg = p.swap ? nseg : 2, s_seg = p.swap ? 2 : nseg;
      int batch = 0;
      for (Walk<OP, PAIR, KEEP> u(p); u.left > 0 && alive; u.next()) {
        const int steps = u.steps(), n0 = u.first_column();
        const int gx = p.swap ? n0 : u.m0, sx = p.swap ? u.m0 : n0;
        for (int k = 0; k < steps; ++k) {
          constexpr int kBatchSteps = kBatch / kStep;
          const int in_batch = k % kBatchSteps;
          if (in_batch == 0) alive = mbar_wait_all(smem_u32(&hdr->ids_full[batch & 1]), (batch >> 1) & 1, abort_flag, p.status.word);
          if (!alive) break;
          int tok[kQuads][4], slot_row[kQuads][4];
          const uint32_t ids = table + static_cast<uint32_t>((batch & 1) * kBatch + in_batch * kStep + part * kQuads * 4) * 4u;
          const bool mine = is_mine();
          if (mine) {
#pragma unroll
            for (int q = 0; q < kQuads; ++q) {
              get4(ids + q * 16u, tok[q]);
              if (!p.tma_rows) get4(ids + 2u * kBatch * 4u + q * 16u, slot_row[q]);
            }
          }
          if (in_batch == kBatchSteps - 1 || k + 1 == steps) {                     // this warp has read the batch
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&hdr->ids_empty[batch & 1]));
            ++batch;
          }
          if (mine) wait_free();
          if (!alive) break;
          const uint32_t bar = full0 + at.slot * 8u;
          const uint32_t dst = ring0 + static_cast<uint32_t>(at.slot) * stage_bytes + static_cast<uint32_t>(part * kQuads) * 512u;
          at.next(stages);
          if (mine && elect_one()) {
#pragma unroll
            for (int s = 0; s < 2; ++s)
              if (s < g_seg) {
#pragma unroll
                for (int q = 0; q < kQuads; ++q)
                  tma_gather4_pair(dst + g_dst + s * kSeg + q * 512u, &map_w, gx + s * 64, tok[q][0], tok[q][1], tok[q][2], tok[q][3], bar);
              }
            if (!p.tma_rows) {
#pragma unroll
              for (int s = 0; s < 2; ++s)
                if (s < s_seg) {
#pragma unroll
                  for (int q = 0; q < kQuads; ++q)
                    tma_gather4_pair(dst + s_dst + s * kSeg + q * 512u, &map_rows, sx + s * 64, slot_row[q][0], slot_row[q][1], slot_row[q][2], slot_row[q][3], bar);
                }
            }
          }
        }
      }
    }
    __syncwarp();
  } else if (warp < kProdWarps && has_cp) {
    // =========================== gather producers ===========================
    const char* Rows = static_cast<const char*>(p.Rows);
    const int cc = tid & 7, r0 = tid >> 3;
    const uint32_t rc_dst = static_cast<uint32_t>(r0) * 128u + (static_cast<uint32_t>(cc ^ (r0 & 7)) << 4);
    const long long pitch_c = static_cast<long long>(p.C) * 2;
    Cursor at;
    bool alive = true;
    auto wait_free = [&]() {             // for the stage at `at`; moves on
      if (at.round > 0) alive = mbar_wait_all(smem_u32(&hdr->empty[at.slot]), (at.round - 1) & 1, abort_flag, p.status.word);
      at.next(stages);
    };
    if constexpr (OP != kOpDweight) {
      // The index warps keep the rows of two units in shared memory.  A unit's are read one step ahead, before the copies of the
      // step before it are issued: a read behind a copy waits for it.
      const uint32_t table = smem0 + kDenseHeader + static_cast<uint32_t>(r0) * 4u;
      const int units = Walk<OP, PAIR, KEEP>(p).left, steps = (p.C + kStep - 1) / kStep;
      int row[4];
      auto read_rows = [&](int t) {
        alive = mbar_wait_all(smem_u32(&hdr->ids_full[t & 1]), (t >> 1) & 1, abort_flag, p.status.word);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          asm volatile("ld.shared.b32 %0, [%1];" : "=r"(row[i]) : "r"(table + static_cast<uint32_t>(t & 1) * (kTileM * 4u) + i * 128u) : "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&hdr->ids_empty[t & 1]));
      };
      if (units > 0) read_rows(0);
      for (int t = 0; t < units && alive; ++t) {
        const char* src[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) src[i] = row[i] >= 0 ? Rows + static_cast<long long>(row[i]) * pitch_c + cc * 16 : nullptr;
        for (int k = 0; k < steps; ++k) {
          const int slot = at.slot;
          wait_free();
          if (alive && k + 1 == steps && t + 1 < units) read_rows(t + 1);
          if (!alive) break;
          const uint32_t base = ring0 + static_cast<uint32_t>(slot) * stage_bytes + rc_dst;
          const bool kvalid = k * kStep + cc * 8 < p.C;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const bool v = kvalid && src[i];
            cp_async16(base + i * 4096u, v ? src[i] : Rows, v ? 16u : 0u);
            if (src[i]) src[i] += 128;
          }
          cp_async_mbar_arrive_noinc(smem_u32(&hdr->full[slot]));
        }
      }
    } else {
      // A 64-row tile is walked with a fixed 16-byte chunk per thread: 16 threads per row of the 128-wide operand (4 rows per
      // thread, 16 apart), 4 * RN threads per row of the BN-wide one (RN rows per thread).  Rows are whole multiples of eight
      // apart, so the swizzle of a thread's chunk is the same in all of them.  A warp must not spend more than some 60
      // instructions on a step (two producer warps share a scheduler, and a step is 500-1000 clocks): the counts are template
      // parameters, the products 32-bit.  Generic loops took 390 instructions and twice the kernel's time.
      // The index warps keep the token (and slot) rows of two batches of kBatch contraction rows in shared memory.  A step's ids
      // are read one step ahead, before the copies of the step before it are issued: a read behind a copy waits for it.
      auto run = [&](auto rn_tag, auto swap_tag, auto tma_tag) {
        constexpr int RN = decltype(rn_tag)::value, kBatchSteps = kBatch / kStep;
        constexpr bool SWAP = decltype(swap_tag)::value, TMA = decltype(tma_tag)::value;
        constexpr int RG = SWAP ? RN : 4, RS = SWAP ? 4 : RN;                      // rows per thread: gathered, slot operand
        constexpr int TN = 4 * RN;                                                 // threads per row of the BN-wide operand
        const int m_c = tid & 15, m_r = tid >> 4, n_c = tid & (TN - 1), n_r = tid / TN;
        const bool n_on = n_c * 8 < p.half;
        const int g_c = SWAP ? n_c : m_c, g_r = SWAP ? n_r : m_r, s_c = SWAP ? m_c : n_c, s_r = SWAP ? m_r : n_r;
        const bool g_on = !SWAP || n_on, s_on = !TMA && (SWAP || n_on);
        constexpr uint32_t GSTEP = kStep / RG, SSTEP = kStep / RS;                 // rows from one of a thread's copies to the next
        const uint32_t g_dst = ring0 + (SWAP ? kMTile : 0u) + static_cast<uint32_t>(g_c >> 3) * kSeg + g_r * 128u + (((g_c & 7) ^ (g_r & 7)) << 4);
        const uint32_t s_dst = ring0 + (SWAP ? 0u : kMTile) + static_cast<uint32_t>(s_c >> 3) * kSeg + s_r * 128u + (((s_c & 7) ^ (s_r & 7)) << 4);
        const unsigned g_pitch = static_cast<unsigned>(SWAP ? p.N : p.C) * 2u, s_pitch = static_cast<unsigned>(SWAP ? p.C : p.N) * 2u;
        const uint32_t table = smem0 + kDenseHeader;                               // [2][token][kBatch], then [2][slot][kBatch]
        auto get = [](uint32_t a) -> int {
          int v;
          asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
          return v;
        };
        int tg[RG], ts[RS];
        auto read_ids = [&](uint32_t at) {             // the ids of one step: its first entry in the token table
#pragma unroll
          for (int j = 0; j < RG; ++j) tg[j] = get(at + (g_r + j * GSTEP) * 4u);
          if (!TMA) {
#pragma unroll
            for (int j = 0; j < RS; ++j) ts[j] = get(at + 2u * kBatch * 4u + (s_r + j * SSTEP) * 4u);
          }
        };
        int batch = 0;                                                             // batches begun by this CTA
        Walk<OP, PAIR, KEEP> u(p);
        if (u.left > 0) {
          alive = mbar_wait_all(smem_u32(&hdr->ids_full[0]), 0u, abort_flag, p.status.word);
          read_ids(table);
        }
        for (; u.left > 0 && alive; u.next()) {
          const int steps = u.steps();
          const int nc0 = u.first_column();
          const int f0 = (SWAP ? nc0 : u.m0) + g_c * 8, s0 = (SWAP ? u.m0 : nc0) + s_c * 8;       // first feature of the chunk
          const bool g_in = f0 < (SWAP ? p.N : p.C), s_in = s0 < (SWAP ? p.C : p.N);
          const char* g_col = Rows + (g_in ? static_cast<long long>(f0) * 2 : 0ll);
          const char* s_col = static_cast<const char*>(p.Slot) + (s_in ? static_cast<long long>(s0) * 2 : 0ll);
          for (int k = 0; k < steps; ++k) {
            const int slot = at.slot;
            wait_free();
            if (!alive) break;
            int cg[RG], cs[RS];
#pragma unroll
            for (int j = 0; j < RG; ++j) cg[j] = tg[j];
            if (!TMA) {
#pragma unroll
              for (int j = 0; j < RS; ++j) cs[j] = ts[j];
            }
            const bool unit_end = k + 1 == steps;
            if (!unit_end && (k + 1) % kBatchSteps != 0) {
              read_ids(table + static_cast<uint32_t>(batch & 1) * (kBatch * 4u) + static_cast<uint32_t>((k + 1) % kBatchSteps) * (kStep * 4u));
            } else {                                   // the next batch: of this unit or of the next one
              __syncwarp();
              if (lane == 0) mbar_arrive(smem_u32(&hdr->ids_empty[batch & 1]));    // this warp has read the batch
              ++batch;
              if (!unit_end || u.left > 1) {
                alive = mbar_wait_all(smem_u32(&hdr->ids_full[batch & 1]), (batch >> 1) & 1, abort_flag, p.status.word);
                if (!alive) break;
                read_ids(table + static_cast<uint32_t>(batch & 1) * (kBatch * 4u));
              }
            }
            const uint32_t base = static_cast<uint32_t>(slot) * stage_bytes;
            if (g_on && (RG > 1 || g_r < kStep)) {
#pragma unroll
              for (int j = 0; j < RG; ++j)
                cp_async16(base + g_dst + j * GSTEP * 128u, g_col + static_cast<unsigned long long>(static_cast<unsigned>(max(cg[j], 0))) * g_pitch,
                           (g_in && cg[j] >= 0) ? 16u : 0u);
            }
            if (s_on && (RS > 1 || s_r < kStep)) {
#pragma unroll
              for (int j = 0; j < RS; ++j)
                cp_async16(base + s_dst + j * SSTEP * 128u, s_col + static_cast<unsigned long long>(static_cast<unsigned>(max(cs[j], 0))) * s_pitch,
                           (s_in && cs[j] >= 0) ? 16u : 0u);
            }
            cp_async_mbar_arrive_noinc(smem_u32(&hdr->full[slot]));
          }
        }
      };
      auto pick_rn = [&](auto swap_tag, auto tma_tag) {
        if (p.half > 128) run(std::integral_constant<int, 8>{}, swap_tag, tma_tag);
        else if (p.half > 64) run(std::integral_constant<int, 4>{}, swap_tag, tma_tag);
        else if (p.half > 32) run(std::integral_constant<int, 2>{}, swap_tag, tma_tag);
        else run(std::integral_constant<int, 1>{}, swap_tag, tma_tag);
      };
      if (p.swap) {
        if (p.tma_rows) pick_rn(std::true_type{}, std::true_type{});
        else pick_rn(std::true_type{}, std::false_type{});
      } else {
        if (p.tma_rows) pick_rn(std::false_type{}, std::true_type{});
        else pick_rn(std::false_type{}, std::false_type{});
      }
    }
    cp_async_wait_all();
  } else if (warp < kMmaWarp) {
    if (warp >= kProdWarps || readers > kEpiWarps) {
    // =========================== read-out ===========================
    const int ew = warp >= kProdWarps ? warp - kProdWarps : warp + kEpiWarps;
    const int lg = ew & 3, share = ew >> 2, shares = readers >> 2;       // TMEM lane group (warp number mod 4), share of the column blocks
    const uint32_t area = epi0 + static_cast<uint32_t>(ew) * 4096u;
    const uint32_t lane_base = static_cast<uint32_t>(lg * 32) << 16;
    T* out = static_cast<T*>(p.Out);
    bool alive = true;
    pdl_wait();                                          // zeros the results are added to, the scatter's plan
    const bool f32_rows = OP == kOpScatter && p.plan[kPlanHot] != 0;
    int t = 0;
    for (Walk<OP, PAIR, KEEP> u(p); u.left > 0 && alive; u.next(), ++t) {
      const int bn = min(Walk<OP, PAIR, KEEP>::kTails ? u.bn : p.BN, p.N - u.n0);              // columns of this tile (a multiple of 8)
      const int n_end = u.n0 + bn;
      int my_ro = -1;                                    // G, S: destination row of tile row lg * 32 + lane
      if (OP != kOpDweight) {
        alive = mbar_wait_all(smem_u32(&hdr->dst_full[t & 1]), (t >> 1) & 1, abort_flag, p.status.word);
        if (!alive) break;
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(my_ro)
                     : "r"(smem0 + kDenseHeader + static_cast<uint32_t>((2 + (t & 1)) * kTileM + lg * 32 + lane) * 4u) : "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&hdr->dst_empty[t & 1]));
      }
      const T* bias_row = (OP != kOpDweight && p.bias) ? static_cast<const T*>(p.bias) + static_cast<long long>(u.e) * p.N + u.n0 : nullptr;
      const int buf = t & 1;
      alive = mbar_wait_all(smem_u32(&hdr->acc_full[buf]), (t >> 1) & 1, abort_flag, p.status.word);
      if (!alive) break;
      tc_fence_after();
      const uint32_t acc = tmem_base + lane_base + static_cast<uint32_t>(buf) * acc_cols;
      bool released = false;
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (PAIR) mbar_arrive_cluster_relaxed(map_to_cta(smem_u32(&hdr->acc_empty[buf]), 0));
          else mbar_arrive(smem_u32(&hdr->acc_empty[buf]));
        }
        released = true;
      };
      const bool packed = OP == kOpGather || (OP == kOpScatter && !f32_rows) || (OP == kOpDweight && p.splits == 1 && p.lane_rows);
      if (packed) {
        // 64 columns = 128 bytes of a 16-bit row at a time, eight lanes to a row: S adds 16 bytes a lane (the memory system takes
        // 39 KB a microsecond from an SM that way).  Bulk reductions of 128 bytes, one per row and lane, took 85 clocks each to
        // issue: 9000 clocks a 128 x 256 tile against 3800 of a contraction of 256.
        for (int c = share; c * 64 < bn; c += shares) {
          const uint32_t srow = area + static_cast<uint32_t>(lane) * 128u;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (c * 64 + h * 32 < bn) {
              uint32_t v[32];
              tmem_ld32(acc + static_cast<uint32_t>(c * 64 + h * 32), v);
              tmem_ld_wait();
              if (OP != kOpDweight && bias_row) add_bias32<T>(bias_row + c * 64 + h * 32, bn - (c * 64 + h * 32), v);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const int ch = h * 4 + j;
                asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(
                                 srow + static_cast<uint32_t>(ch ^ (lane & 7)) * 16u),
                             "r"(pack2(out, v[8 * j], v[8 * j + 1])), "r"(pack2(out, v[8 * j + 2], v[8 * j + 3])),
                             "r"(pack2(out, v[8 * j + 4], v[8 * j + 5])), "r"(pack2(out, v[8 * j + 6], v[8 * j + 7]))
                             : "memory");
              }
            }
          }
          if ((c + shares) * 64 >= bn) release();        // the accumulator has been read: the next tile but one may begin
          const int col0 = u.n0 + c * 64;
          __syncwarp();
          const int j = lane & 7, col = col0 + j * 8;
          uint4 x[8];
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int row = it * 4 + (lane >> 3);
            asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];"
                         : "=r"(x[it].x), "=r"(x[it].y), "=r"(x[it].z), "=r"(x[it].w)
                         : "r"(area + row * 128u + (static_cast<uint32_t>(j ^ (row & 7)) << 4))
                         : "memory");
          }
          __syncwarp();
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int row = it * 4 + (lane >> 3);
            long long ro;
            if (OP != kOpDweight) {
              ro = __shfl_sync(0xffffffffu, my_ro, row);
            } else {
              const int f = u.m0 + lg * 32 + row;
              ro = f < p.C ? static_cast<long long>(u.e) * p.C + f : -1;
            }
            if (ro >= 0 && col < n_end) {
              if (OP == kOpScatter) red8(out + ro * p.N + col, x[it]);
              else *reinterpret_cast<uint4*>(out + ro * p.N + col) = x[it];
            }
          }
        }
      } else {
        for (int c = share; c * 32 < bn; c += shares) {
          const int col0 = u.n0 + c * 32;
          uint32_t v[32];
          tmem_ld32(acc + static_cast<uint32_t>(c * 32), v);
          tmem_ld_wait();
          if (OP == kOpScatter) {
            warp_regs_emit(v, area, lane, [&](int row, int cj, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3) {
              const int ro = __shfl_sync(0xffffffffu, my_ro, row);
              const int col = col0 + cj;
              if (ro >= 0 && col < n_end) {
                const long long off = static_cast<long long>(ro) * p.N + col;
                if (bias_row) add_bias4<T>(bias_row + c * 32 + cj, x0, x1, x2, x3);
                red4(p.acc + off, x0, x1, x2, x3);
              }
            });
          } else if (OP == kOpDweight && p.lane_rows) {  // partial sums, output rows = accumulator rows
            warp_regs_emit(v, area, lane, [&](int row, int cj, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3) {
              const int f = u.m0 + lg * 32 + row, col = col0 + cj;
              if (f < p.C && col < n_end) red4(p.acc + (static_cast<long long>(u.e) * p.C + f) * p.N + col, x0, x1, x2, x3);
            });
          } else if (OP == kOpDweight) {                 // output rows = accumulator columns
            warp_cols_emit(v, area, lane, [&](int ci, int f4, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3) {
              const int f = u.m0 + lg * 32 + f4;
              if (f < p.C && col0 + ci < n_end) {
                const long long off = (static_cast<long long>(u.e) * p.N + col0 + ci) * p.C + f;
                if (p.splits > 1) red4(p.acc + off, x0, x1, x2, x3);
                else store4(out + off, x0, x1, x2, x3);
              }
            });
          }
        }
      }
      if (!released) release();
    }
    if (OP == kOpScatter && !KEEP && f32_rows && p.rounds) {
      __threadfence();                                   // (before the barrier of the common exit: what this thread has added)
      if (tid == kProdThreads) hdr->rounds = 1;
    }
    }
  } else if (warp == kMmaWarp) {
    // =========================== MMA issuer ===========================
    if (leader) {
      const bool a_mn = OP == kOpDweight, b_mn = OP == kOpDweight || !p.nc;
      const uint64_t a_desc = a_mn ? make_smem_desc(0u, kSeg, 1024u) : make_smem_desc(0u, 16u, 1024u);
      const uint64_t b_desc = (b_mn ? make_smem_desc(0u, kSeg, 1024u) : make_smem_desc(0u, 16u, 1024u)) + (kMTile >> 4);
      const uint32_t a_adv = (a_mn ? 16u * 128u : 32u) >> 4, b_adv = (b_mn ? 16u * 128u : 32u) >> 4;
      bool ok = true;
      int t = 0, a_first = 0, a_next = 0;                // slots of the row block's first tile and of the tile after its last
      Cursor at;
      for (Walk<OP, PAIR, KEEP> u(p); u.left > 0 && ok; u.next(), ++t) {
        const int steps = u.steps();
        if (KEEP && u.j == 0) a_first = a_next;
        a_next = a_first;
        const uint32_t idesc =
            make_idesc(Elem<T>::fmt, a_mn ? 1u : 0u, b_mn ? 1u : 0u, PAIR ? 2 * kTileM : kTileM, static_cast<uint32_t>(u.width()));
        const int buf = t & 1;
        if (t >= 2) {
          ok = mbar_wait_all<PAIR>(smem_u32(&hdr->acc_empty[buf]), ((t >> 1) - 1) & 1, abort_flag, p.status.word);
          if (!ok) break;
        }
        const uint32_t d = tmem_base + static_cast<uint32_t>(buf) * acc_cols;
        for (int ks = 0; ks < steps; ++ks) {
          ok = mbar_wait_all<PAIR>(smem_u32(&hdr->full[at.slot]), at.round & 1, abort_flag, p.status.word);
          if (!ok) break;
          if (has_cp) fence_proxy_async_smem();
          const uint32_t empty = smem_u32(&hdr->empty[at.slot]);
          // (descriptors: 14 address bits in 16-byte units; shared memory is smaller)
          const uint32_t addr = (ring0 + static_cast<uint32_t>(at.slot) * stage_bytes) >> 4;
          const uint32_t a_addr = KEEP ? a_tile(a_next) >> 4 : addr;
          if (KEEP && ++a_next == p.a_slots) a_next = 0;
          at.next(stages);
          tc_fence_after();
          if (elect_one()) {
            umma_f16_x4<PAIR>(d, a_desc + a_addr, b_desc + addr, a_adv, b_adv, idesc, ks > 0 ? 1u : 0u);
            umma_done<PAIR>(empty);
            if (ks + 1 == steps) umma_done<PAIR>(smem_u32(&hdr->acc_full[buf]));
          }
        }
      }
    }
    pdl_trigger();                       // (not before: a dependent's waiting CTAs would keep a kernel of another stream off this SM)
    __syncwarp();
  } else if (warp >= kIndexWarp) {
    // =========================== index warps ===========================
    const uint32_t table = smem0 + kDenseHeader;
    const int it = tid - kIndexWarp * 32;
    bool alive = true;
    if constexpr (OP != kOpDweight) {
      // the first warp: where the producers find the rows; the second: where the read-out puts them
      const bool dst = warp != kIndexWarp;
      unsigned long long* full = dst ? hdr->dst_full : hdr->ids_full;
      unsigned long long* empty = dst ? hdr->dst_empty : hdr->ids_empty;
      int t = 0;
      for (Walk<OP, PAIR, KEEP> u(p); (dst || gathers) && u.left > 0 && alive; u.next(), ++t) {
        int row[4], b[4];
        long long id[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int m = u.m0 + lane + 32 * i;
          b[i] = p.by_k.quotient(m);
          row[i] = m < p.M ? (b[i] * p.E + u.e) * p.K + (m - b[i] * p.K) : -1;
          id[i] = (row[i] >= 0 && (dst || OP == kOpGather)) ? load_index(p.Ind, p.index_dtype, row[i]) : 0;
        }
        if (t >= 2) alive = mbar_wait_all(smem_u32(&empty[t & 1]), ((t >> 1) - 1) & 1, abort_flag, p.status.word);
        if (!alive) break;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const bool known = row[i] >= 0 && id[i] >= 0 && id[i] < p.T;
          const int token_row = b[i] * p.T + static_cast<int>(id[i]);
          int v;
          if (!dst) {
            v = OP == kOpScatter ? row[i] : (known ? token_row : -1);
          } else {
            if (row[i] >= 0 && !known && u.n0 == 0) p.status.report(EGS_STATUS_INDEX_OUT_OF_RANGE);
            v = OP == kOpGather ? row[i] : known ? token_row : -1;
          }
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(table + static_cast<uint32_t>(((dst ? 2 : 0) + (t & 1)) * kTileM + lane + 32 * i) * 4u), "r"(v) : "memory");
        }
        mbar_arrive(smem_u32(&full[t & 1]));
      }
    } else {
      constexpr int kPer = kBatch / (kIndexWarps * 32);
      int batch = 0;
      for (Walk<OP, PAIR, KEEP> u(p); u.left > 0 && alive; u.next()) {
        const int m_begin = u.split * p.rows_per_split, m_end = min(p.M, m_begin + p.rows_per_split);
        const bool report = u.m0 == 0 && u.n0 == 0;
        for (int m0 = m_begin; m0 < m_end && alive; m0 += kBatch, ++batch) {
          int tok[kPer], slot_row[kPer];
          long long t[kPer];
#pragma unroll
          for (int i = 0; i < kPer; ++i) {                 // all loads first
            const int m = m0 + it + i * kIndexWarps * 32;
            const bool on = m < m_end;
            tok[i] = on ? p.by_k.quotient(m) : 0;
            const int s = (tok[i] * p.E + u.e) * p.K + (on ? m - tok[i] * p.K : 0);
            t[i] = load_index(p.Ind, p.index_dtype, s);
            slot_row[i] = on ? s : -1;
          }
#pragma unroll
          for (int i = 0; i < kPer; ++i) {
            const bool known = t[i] >= 0 && t[i] < p.T;
            if (slot_row[i] >= 0 && !known && report) p.status.report(EGS_STATUS_INDEX_OUT_OF_RANGE);
            tok[i] = (slot_row[i] >= 0 && known) ? tok[i] * p.T + static_cast<int>(t[i]) : -1;
          }
          if (batch >= 2) alive = mbar_wait_all(smem_u32(&hdr->ids_empty[batch & 1]), ((batch >> 1) - 1) & 1, abort_flag, p.status.word);
          if (!alive) break;
          const uint32_t dst = table + static_cast<uint32_t>(batch & 1) * (kBatch * 4u) + static_cast<uint32_t>(it) * 4u;
#pragma unroll
          for (int i = 0; i < kPer; ++i) {
            asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + i * kIndexWarps * 128u), "r"(tok[i]) : "memory");
            if (!p.tma_rows) asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + 2u * kBatch * 4u + i * kIndexWarps * 128u), "r"(slot_row[i]) : "memory");
          }
          mbar_arrive(smem_u32(&hdr->ids_full[batch & 1]));
        }
      }
    }
  } else if (has_tma) {
    // =========================== TMA issuer ===========================
    // a pair's stage is announced by the leader, for both CTAs and for what the producers gather
    const uint32_t bytes = PAIR ? 2u * stage_bytes : (OP != kOpDweight ? n_bytes : (p.swap ? kMTile : n_bytes)) + ((OP == kOpScatter && p.tma_rows) ? kMTile : 0u);
    bool ok = true;
    int a_slot = 0;
    uint32_t n = 0;                      // steps before this tile
    auto tell_reached = [&]() {
      if (gathers && lane == 0) asm volatile("st.release.cta.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&hdr->reached)), "r"(n) : "memory");
    };
    Cursor at;
    for (Walk<OP, PAIR, KEEP> u(p); u.left > 0 && ok; u.next()) {
      const int steps = u.steps();
      const int n0 = u.first_column();
      const int column = OP == kOpDweight && p.swap ? u.m0 : n0, x0 = p.whole ? 0 : column, z0 = p.whole ? column >> 6 : 0;
      const bool rows_too = !KEEP || u.j == 0;       // a scatter's row block is loaded with its first column tile
      // (a half tile's columns come in boxes of a whole one where those are of whole segments or of weights [E, N, C]: the MMAs do not read the rest)
      const bool less = Walk<OP, PAIR, KEEP>::kTails && u.bn < p.BN && !p.whole && !p.nc;
      const int boxes = less ? u.segs() : p.boxes;
      const uint32_t unit_bytes = less ? 2u * (kMTile + static_cast<uint32_t>(u.segs()) * kSeg) : bytes;
      int m = OP == kOpDweight ? u.split * p.rows_per_split : u.m0;
      int b = p.by_k.quotient(m), k = m - b * p.K;     // first slot row of the step
      if (KEEP) {
        if (u.j == 0) tell_reached();
        n += steps;
      }
      for (int ks = 0, c0 = 0; ks < steps; ++ks, c0 += kStep) {
        if (at.round > 0) {
          ok = mbar_wait_all(smem_u32(&hdr->empty[at.slot]), (at.round - 1) & 1, abort_flag, p.status.word);
          if (!ok) break;
        }
        const uint32_t own = smem_u32(&hdr->full[at.slot]), base = ring0 + static_cast<uint32_t>(at.slot) * stage_bytes;
        const uint32_t bar = PAIR ? map_to_cta(own, 0) : own;
        at.next(stages);
        auto box3 = [&](uint32_t dst, int x, int y) {
          if (PAIR) tma_load_3d_pair(dst, &map_w, x, y, u.e, bar);
          else tma_load_3d(dst, &map_w, x, y, u.e, bar);
        };
        auto box4 = [&](uint32_t dst, int x) {
          if (PAIR) tma_load_4d_pair(dst, &map_rows, x, k, u.e, b, bar);
          else tma_load_4d(dst, &map_rows, x, k, u.e, b, bar);
        };
        if (elect_one()) {
          if (leader) mbar_arrive_expect_tx(own, rows_too ? unit_bytes : (PAIR ? 2u : 1u) * n_bytes);
          if (OP != kOpDweight) {
            if (OP == kOpScatter && p.tma_rows && rows_too) box4(KEEP ? a_tile(a_slot) : base, c0);
            if (p.nc) {
              box3(base + kMTile, c0, n0);
            } else {
#pragma unroll
              for (int s = 0; s < 4; ++s)
                if (s < boxes) {
                  if (PAIR) tma_load_4d_pair(base + kMTile + s * kSeg, &map_w, x0 + s * 64, c0, z0, u.e, bar);
                  else tma_load_4d(base + kMTile + s * kSeg, &map_w, x0 + s * 64, c0, z0, u.e, bar);
                }
            }
          } else if (p.tma_rows) {
            const uint32_t dst = base + (p.swap ? 0u : kMTile);
#pragma unroll
            for (int s = 0; s < 4; ++s)
              if (s < boxes) tma_load_5d<PAIR>(dst + s * kSeg, &map_rows, x0 + s * 64, k, b, z0, u.e, bar);
          }
        }
        if (KEEP && rows_too && ++a_slot == p.a_slots) a_slot = 0;
        if (OP == kOpDweight) {
          k += kStep;                                  // 64 rows are parts of one batch element or whole ones
          while (k >= p.K) { k -= p.K; ++b; }
        }
      }
    }
    if (KEEP && ok) tell_reached();
    __syncwarp();
  }

  // ---- common exit ----
  tc_fence_before();
  __syncthreads();
  if (OP == kOpScatter && !KEEP && hdr->rounds && *abort_flag == 0u) round_rows<T, PAIR>(p, hdr);
  if (!PAIR) {
    if (warp == kMmaWarp) tmem_release(tmem_base, tmem_cols, smem_u32(&hdr->drain), abort_flag, p.status, lane);
  } else {
    // nobody leaves while the partner may still read its shared memory, write its tensor memory or signal its barriers; after an
    // abort MMAs of the pair may still be in flight, and the leader waits for them (bounded) before the pair meets
    uint32_t safe = 1u;
    if (warp == kMmaWarp && *abort_flag) {
      if (lane == 0) {
        uint32_t ignore_abort = 0u;
        p.status.tell_host();
        umma2_commit(smem_u32(&hdr->drain));
        safe = mbar_wait(smem_u32(&hdr->drain), 0u, &ignore_abort, nullptr) ? 1u : 0u;
      }
      safe = __shfl_sync(0xffffffffu, safe, 0);
    }
    cluster_sync_all();
    if (warp == kMmaWarp && safe) {
      tc_fence_after();
      tmem_dealloc2(tmem_base, tmem_cols);
    }
  }
}

// Slot rows can come as one TMA box per 64-element column segment when `rows` consecutive expert rows starting at a multiple of
// `rows` are whole batch elements or lie inside one.
bool rows_fit_boxes(int K, int rows) { return K % rows == 0 || rows % K == 0; }
// The same rows one by one, for tile::gather4: rows of 64 elements of a [rows, width] matrix.
bool encode_gather(TensorMap3* map, const void* base, long long rows, int width) {
  const unsigned long long dims[2] = {static_cast<unsigned long long>(width), static_cast<unsigned long long>(rows)};
  const unsigned box[2] = {64u, 1u};
  return encode_tensor_map_16bit(map, base, 2, dims, box);
}
bool encode_slot_rows(TensorMap3* map, const void* base, int B, int E, int K, int width, int rows) {
  const unsigned kk = static_cast<unsigned>(K < rows ? K : rows);
  const unsigned long long dims[4] = {static_cast<unsigned long long>(width), static_cast<unsigned long long>(K),
                                      static_cast<unsigned long long>(E), static_cast<unsigned long long>(B)};
  const unsigned box[4] = {64u, kk, 1u, static_cast<unsigned>(rows) / kk};
  return encode_tensor_map_16bit(map, base, 4, dims, box);
}

// A tile whose rows are contraction elements comes 64 columns at a time, which is as wide as a swizzled box gets.  Seen as [rows, 64] matrices
// side by side, the segments of a tile are one box of several of them, where segments are whole and a CTA's columns begin with one: one
// load instead of two or four (bf16, G of 262144 rows of 64 experts, 1024 -> 256 features 114 -> 109 us, of 65536 rows, 2048 -> 512 104 -> 101).
bool whole_segments(int width, int staged, bool pair) { return staged % 64 == 0 && width % (pair ? 128 : 64) == 0; }

// One CTA per tile of 128 x BN or a pair of CTAs per tile of 256 x BN, and BN, by clocks.  A step writes and reads 128 + `staged`
// rows of 128 bytes of a CTA's shared memory, 2 clocks a row at 128 bytes a clock (measured: 2.0 in pairs, 2.4 on single CTAs, 2.6 for
// their scatters), the tensor core multiplies BN columns in 2 * BN clocks, the load/store unit needs lsu0 + lsu1 * staged for its
// share of the copies, and the barriers of a step take 600 (800 in a scatter that gathers its rows).  In G the copies of single CTAs, handed over
// by their threads, hold a step up to 750 where there is more than one wave of them, and a pair's gathers beside less than 64 columns to
// 850 (weights [E, N, C]: 750).  With 600 there all of these stayed on single CTAs: 512 rows of 256 experts, 512 -> 128 features, 33.3 us, on
// pairs 30.3; 5724 of 10, 1056 -> 136, 41.5 and 37.4; 4515 of 45, 864 -> 104, 84 and 65.  Of 1600 calls of G, sizes drawn, 174 run otherwise than with 600
// and take 0.91 of the time in the mean; the slowest 1.08 (1292 rows of 109 experts, 328 -> 280, on pairs), 1.06 (2400 of 12, 152 -> 304, tiles of 160, not
// 112) and 1.05 (1085 of 20, 704 -> 88).  Widths that are held up alike cost the same here, but more columns still take longer: of those
// that need as many waves only the narrowest is looked at (133 experts of 296 rows, 1432 -> 280: 80.8 us with tiles of 144, 88.2 with 176).
// Read-out takes epi clocks a
// column beside the next tile's main loop; the additions of a scatter share the way to the L2 with the loads, and half of the shorter
// one shows.  Units go out in waves of one per SM or pair of SMs; a pair starts and ends 2500 clocks slower.
//
// The rows of a scatter whose contraction is short enough stay in a pair's shared memory for several column tiles, and the loads hide better
// beside the additions: a fifth of the shorter one shows, not half, or 0.3 of it where only four stages are left.  (B=512 as above, S
// without its fill: nothing taken out 1285 us, rows loaded for the first column tile only 1115, no loads 820, no additions 840.)
// They stay where the estimate gains 2 % over single CTAs, whose gathers it takes for faster than they are, and 4 % over pairs.  Both
// forms were measured for 159 sizes (bf16, whole calls, against rows loaded for every column tile): the 134 that stay take 0.966 of
// the time in the median, a quarter 0.77 to 0.93, ten 1.03 to 1.07 - seven of those have weights beyond 64 MB and token rows beyond the L2,
// where 0.94 to 1.07 came out, 0.99 in the mean; of the others one would gain 6 %, three 4 %.  All together 0.960 of the time; 0.965
// with one margin of 5.5 % and no difference for four stages, 0.955 if every size took what is faster.
struct Ring {
  int stages = 0, a_slots = 0, readers = kEpiWarps;
};
struct Tile {
  int bn = 256;
  int group = 0, full_waves = 0;         // see Walk; 0: nothing stays
  bool pair = false;
  double cost = 1e30;
};
size_t column_bytes(int half, bool nc_tile) { return nc_tile ? static_cast<size_t>(half) * 128 : static_cast<size_t>((half + 63) / 64) * kSeg; }
// stages, with room for `keep` tiles of the 128-wide operand, in what `not_ring` bytes leave
Ring fit_ring(int half, bool nc_tile, size_t not_ring, int keep) {
  Ring r;
  for (int s = kMaxStages; s > 0 && r.stages == 0; --s) {
    const int slots = s > keep ? s : keep;
    if (not_ring + slots * kMTile + s * column_bytes(half, nc_tile) <= kSmemMax) {
      r.stages = s;
      r.a_slots = slots;
    }
  }
  return r;
}
// S: sixteen read-out warps where nothing is gathered; eight where their room is wanted for the rows that stay.  At least four stages,
// or the rows cannot stay (stages = 0).  (On single CTAs, which stage twice the columns, rows that stayed gained nothing.)
Ring fit_scatter(int half, bool nc_tile, bool boxes, int keep) {
  const size_t fixed = kDenseHeader + kRowTable;
  Ring r = fit_ring(half, nc_tile, fixed + epi_bytes(boxes), keep);
  if (boxes) r.readers = kProdWarps + kEpiWarps;
  if (keep == 0 || r.stages >= 4) return r;
  if (boxes) r = fit_ring(half, nc_tile, fixed + epi_bytes(false), keep);
  if (r.stages < 4) r.stages = 0;
  return r;
}
Tile pick_tile(int n, int m, long long groups, int steps, double lsu0, double lsu1, double epi, bool scatter, bool nc_tile = false, bool gather = false) {
  Tile best, stay;                       // units of one tile; rows that stay
  for (int pair = 0; pair < 2; ++pair) {
    const int rows = pair ? 2 * kTileM : kTileM, sms = pair ? kSms / 2 : kSms, unit16 = pair ? 32 : 16;
    const double per_row = pair ? 2.0 : scatter ? 2.6 : 2.4;
    const long long row_units = (m + rows - 1) / rows * groups;
    const int top = n < 256 ? (n + unit16 - 1) / unit16 * unit16 : 256;
    const bool boxes = lsu0 == 0.0;
    for (int bn = top; bn >= unit16; bn -= unit16) {
      const long long tiles = (n + bn - 1) / bn;
      const int staged = pair ? bn / 2 : bn;
      const long long units = row_units * tiles, waves = (units + sms - 1) / sms;
      if (gather && !pair && waves > 1 && bn > unit16 && (row_units * ((n + bn - unit16 - 1) / (bn - unit16)) + sms - 1) / sms == waves) continue;
      const double least = scatter && lsu0 > 0.0 ? 800.0 : !gather ? 600.0 : pair ? (std::min(bn, n) >= 64 ? 600.0 : nc_tile ? 750.0 : 850.0) : waves > 1 ? 750.0 : 600.0;
      double step = per_row * (128 + staged);
      if (2.0 * bn > step) step = 2.0 * bn;
      if (lsu0 + lsu1 * staged > step) step = lsu0 + lsu1 * staged;
      if (step < least) step = least;
      const double loop = steps * step, out = epi * bn, more = loop > out ? loop : out, less = scatter ? (loop > out ? out : loop) : 0.0;
      const double ends = out + (pair ? 2500 : 0);
      auto consider = [&](Tile& to, double cost, long long group, long long full) {
        if (cost >= to.cost * (pair && !to.pair ? 0.97 : bn != to.bn ? 0.98 : 1.0)) return;
        to.bn = bn;
        to.group = static_cast<int>(group);
        to.full_waves = static_cast<int>(full);
        to.pair = pair != 0;
        to.cost = cost;
      };
      consider(best, waves * (more + 0.5 * less + 1000) + ends, 0, 0);
      // Rows that stay: whole waves of row blocks, and the rest in one to eight units a row block.  At best that is as if all tiles
      // were spread evenly, which most widths need not be looked at further for.
      if (!scatter || pair == 0 || tiles == 1 || waves * (more + 0.2 * less + 1000) + ends >= 0.98 * stay.cost) continue;
      const Ring ring = fit_scatter(staged, nc_tile, boxes, steps);
      if (ring.stages == 0) continue;
      const double shown = ring.stages == 4 ? 0.3 : 0.2;
      auto tile_cost = [&](long long kept) { return more + (shown + 0.3 / kept) * less + 1000; };
      const long long full = row_units / sms, rest = row_units - full * sms;
      for (long long per_block = 1; per_block <= std::min(tiles, 8ll); ++per_block) {
        const long long group = (tiles + per_block - 1) / per_block, rest_waves = (rest * ((tiles + group - 1) / group) + sms - 1) / sms;
        consider(stay, full * tiles * tile_cost(tiles) + rest_waves * group * tile_cost(group) + ends, group, full);
      }
    }
  }
  return stay.cost < (best.pair ? 0.96 : 0.98) * best.cost ? stay : best;
}

// What Walk needs to know about the grid; r1 and r2 are set.
void plan_walk(DenseParams& p, bool pair) {
  const int most = pair ? kSms / 2 : kSms;
  p.stride = Div(p.full_waves == 0 && p.units < most ? p.units : most);
  p.by_k = Div(p.K);
  p.by_group = Div(p.groups_n);
  p.by_tiles = Div(p.tiles_n);
  auto digits = [&](int u, int* to) {
    to[0] = u % p.r1.d;
    to[1] = u / p.r1.d % p.r2.d;
    to[2] = u / p.r1.d / p.r2.d;
  };
  digits(p.stride.d, p.step_full);
  p.step[0] = p.stride.d % p.groups_n;
  digits(p.stride.d / p.groups_n, p.step + 1);
}

// G on pairs: where the last wave would leave half of the pairs idle or more, its tiles are cut in two: a step of 128 columns takes 0.72 of the time
// of one of 256, so that 3.46 waves take as long as 3.75, not four.  bf16, 32 experts of 2048 rows, 768 -> 192 features 30.1 -> 28.2 us, 24 of 909,
// 1000 -> 200 25.1 -> 23.0, 20 of 1024, 768 -> 512 25.1 -> 23.0.  D, which runs beside the dX / dY kernel and leaves it the idle pairs, keeps whole
// tiles: alone 35.3 -> 33.3 us, but a training step of ragged sizes 139.5 -> 142.
struct Tail {
  int full_waves = 0, units = 0, first = 0;      // units of half a tile, columns of the first half
};
Tail plan_tail(int units, int bn, int n, bool whole) {
  const int pairs = kSms / 2, rest = units % pairs, first = (bn / 2 + 31) / 32 * 32, last = n - (n - 1) / bn * bn;
  Tail t;
  if (units < pairs || rest == 0 || 2 * rest > pairs || bn < 128 || last <= first || (whole && first % 128 != 0)) return t;
  t.full_waves = units / pairs;
  t.units = 2 * rest;
  t.first = first;
  return t;
}

template <typename T, int OP, bool PAIR, bool KEEP>
cudaError_t launch(const DenseParams& p, const TensorMap3& mw, const TensorMap3& mr, cudaStream_t st) {
  const size_t smem = kDenseHeader + (OP == kOpDweight ? table_bytes(!p.tma_rows) : kRowTable) + epi_bytes(p.readers > kEpiWarps) +
                      p.a_slots * kMTile + p.stages * column_bytes(p.half, OP != kOpDweight && p.nc);
  cudaError_t err = ensure_smem_optin<dense16_kernel<T, OP, PAIR, KEEP>>(static_cast<int>(kSmemMax));
  if (err != cudaSuccess) return err;
  const int grid = (PAIR ? 2 : 1) * p.stride.d;
  err = launch_kernel(dense16_kernel<T, OP, PAIR, KEEP>, grid, kDenseThreads, smem, st, true, p, mw, mr);
  count_launch();
  return err;
}
template <int OP, bool PAIR, bool KEEP = false>
cudaError_t launch_typed(const DenseParams& p, int dtype, const TensorMap3& mw, const TensorMap3& mr, cudaStream_t st) {
  return dtype == EGS_F16 ? launch<__half, OP, PAIR, KEEP>(p, mw, mr, st) : launch<__nv_bfloat16, OP, PAIR, KEEP>(p, mw, mr, st);
}

}  // namespace

void configure_dense16_rowgemm(RowGemmParams& p, bool scatter) {
  const int steps = (p.C + kStep - 1) / kStep;
  const bool cp_rows = !scatter || !rows_fit_boxes(p.K, 128);
  const bool nc = p.w_layout == EGS_W_NC;
  const Tile t = pick_tile(p.N, p.M, p.E, steps, cp_rows ? 340.0 : 0.0, 0.0, 16.0, scatter, nc, !scatter);
  p.BN = t.bn;
  p.pair = t.pair ? 1 : 0;
  p.tile_group = t.group;
  p.full_waves = t.full_waves;
  p.slot_boxes = scatter && !cp_rows ? 1 : 0;
  const Ring r = fit_scatter(p.pair ? p.BN / 2 : p.BN, nc, p.slot_boxes != 0, t.group > 0 ? steps : 0);
  p.stages = r.stages;
  p.row_tiles = 1;
  p.persistent = 1;
}

void dense16_half_tiles(const RowGemmParams& r, int* units, int* first) {
  *units = *first = 0;
  if (!r.pair) return;
  const long long all = static_cast<long long>((r.M + 2 * kTileM - 1) / (2 * kTileM)) * ((r.N + r.BN - 1) / r.BN) * r.E;
  if (all > 2147483647ll - kSms) return;
  const Tail t = plan_tail(static_cast<int>(all), r.BN, r.N, r.w_layout != EGS_W_NC && whole_segments(r.N, r.BN / 2, true));
  *units = t.units;
  *first = t.first;
}

cudaError_t launch_dense16_rowgemm(const RowGemmParams& r, bool scatter, int dtype, cudaStream_t st) {
  DenseParams p{};
  p.Rows = r.A; p.bias = r.bias; p.Ind = r.Ind; p.Out = r.Out; p.acc = r.acc; p.plan = r.plan; p.rounds = r.rounds; p.status = r.status;
  p.B = r.B; p.T = r.T; p.E = r.E; p.K = r.K; p.M = r.M; p.C = r.C; p.N = r.N;
  p.nc = r.w_layout == EGS_W_NC;
  p.index_dtype = r.index_dtype;
  p.BN = r.BN; p.stages = r.stages;
  p.half = r.pair ? r.BN / 2 : r.BN;
  p.after_own = r.after_own;
  const int rows = r.pair ? 2 * kTileM : kTileM;
  p.tiles_m = (r.M + rows - 1) / rows;
  p.tiles_n = (r.N + r.BN - 1) / r.BN;
  p.r1 = Div(r.expert_fastest ? 1 : p.tiles_m);
  p.r2 = Div(r.E);
  const Ring ring = fit_scatter(p.half, p.nc != 0, r.slot_boxes != 0, r.tile_group > 0 ? (r.C + kStep - 1) / kStep : 0);
  p.a_slots = ring.a_slots;
  p.readers = ring.readers;
  p.group = r.tile_group > 0 ? r.tile_group : 1;
  p.full_waves = r.full_waves;
  p.groups_n = (p.tiles_n + p.group - 1) / p.group;
  const long long units = static_cast<long long>(p.tiles_m) * p.groups_n * p.E;
  if (units > 2147483647ll - kSms) return cudaErrorInvalidValue;
  p.units = static_cast<int>(units);
  plan_walk(p, r.pair != 0);
  TensorMap3 mw{}, mr{};
  const unsigned long long inner = p.nc ? r.C : r.N, outer = p.nc ? r.N : r.C;
  const unsigned long long dims[3] = {inner, outer, static_cast<unsigned long long>(r.E)};
  const unsigned box[3] = {64u, p.nc ? static_cast<unsigned>(p.half) : static_cast<unsigned>(kStep), 1u};
  if (p.nc) {
    if (!encode_tensor_map_16bit(&mw, r.W, 3, dims, box)) return cudaErrorInvalidValue;
  } else {
    p.whole = whole_segments(r.N, p.half, r.pair != 0);
    p.boxes = p.whole ? 1 : (p.half + 63) / 64;
    const unsigned long long segs[4] = {p.whole ? 64ull : inner, outer, p.whole ? inner / 64 : 1ull, static_cast<unsigned long long>(r.E)};
    const unsigned long long strides[3] = {inner * 2, 128ull, inner * outer * 2};
    const unsigned seg_box[4] = {64u, static_cast<unsigned>(kStep), p.whole ? static_cast<unsigned>(p.half / 64) : 1u, 1u};
    if (!encode_tensor_map_16bit_strided(&mw, r.W, 4, segs, strides, seg_box)) return cudaErrorInvalidValue;
  }
  p.tma_rows = r.slot_boxes;
  if (p.tma_rows && !encode_slot_rows(&mr, r.A, r.B, r.E, r.K, r.C, 128)) return cudaErrorInvalidValue;
  if (r.pair && !p.tma_rows &&
      !encode_gather(&mr, r.A, scatter ? static_cast<long long>(r.M) * r.E : static_cast<long long>(r.B) * r.T, r.C))
    return cudaErrorInvalidValue;
  if (scatter)
    return !r.pair           ? launch_typed<kOpScatter, false>(p, dtype, mw, mr, st)
           : r.tile_group > 0 ? launch_typed<kOpScatter, true, true>(p, dtype, mw, mr, st)
                              : launch_typed<kOpScatter, true>(p, dtype, mw, mr, st);
  if (r.pair) {
    const Tail t = plan_tail(p.units, p.BN, p.N, p.whole != 0);
    if (t.units > 0) p.full_waves = t.full_waves;
    p.tail = t.units;
    p.tail_bn = t.first;
  }
  return r.pair ? launch_typed<kOpGather, true>(p, dtype, mw, mr, st) : launch_typed<kOpGather, false>(p, dtype, mw, mr, st);
}

// Rows one accumulator of D sums: the tensor core truncates as it adds, and the error grows with the number of additions, 1.5e-5 of
// the largest sum after 8192 rows. The ranges of a longer contraction are added by float32 atomics, which round.
constexpr int kMaxRangeRows = 8192;

// D: which operand's features are the accumulator's rows, the tile, and the row ranges.
void configure_dense16_dweight(DWeightParams& p) {
  const bool slot_cp = !rows_fit_boxes(p.K, kStep);
  double best = 1e30;
  const long long steps_all = (p.M + kStep - 1) / kStep;
  const long long least = (p.M + kMaxRangeRows - 1) / kMaxRangeRows, most = std::min(std::max(64ll, least), steps_all);
  // the orientation whose accumulator rows are the output's rows first: its read-out stores whole row segments
  const bool pref = p.out_layout == EGS_DW_DIRECT_ROWS;
  for (int o = 0; o < 2; ++o) {
    const bool sw = o == 0 ? pref : !pref;
    const int mf = sw ? p.FD : p.FG, nf = sw ? p.FG : p.FD;
    // load/store clocks per step: 10 per 512 bytes; the gathered operand always, the slot operand where it has no boxes
    const double lsu0 = (!sw ? 320.0 : 0.0) + (sw && slot_cp ? 320.0 : 0.0), lsu1 = (sw ? 2.5 : 0.0) + (!sw && slot_cp ? 2.5 : 0.0);
    for (long long s = least; s <= most; s = s < 4 ? s + 1 : s + s / 2) {
      const long long sp_steps = (steps_all + s - 1) / s;
      const long long real = (steps_all + sp_steps - 1) / sp_steps;      // ranges of whole steps
      const double epi = real > 1 ? 32.0 : o == 0 ? 16.0 : 20.0;         // (partial tiles are added atomically)
      const Tile t = pick_tile(nf, mf, p.E * real, static_cast<int>(sp_steps), lsu0, lsu1, epi, false);
      double cost = t.cost;
      // more than one range: zero fill and rounding of the float32 sums, two launches and 10 bytes an element
      if (real > 1) cost += 9000 + static_cast<double>(p.E) * p.FG * p.FD * 10 / (148 * 20.0);
      if (cost < best * (o == 0 ? 1.0 : 0.97)) {
        best = cost;
        p.swap = sw ? 1 : 0;
        p.BN = t.bn;
        p.pair = t.pair ? 1 : 0;
        p.splits = static_cast<int>(real);
        p.rows_per_split = static_cast<int>(sp_steps * kStep);
      }
    }
  }
  p.stages = fit_ring(p.pair ? p.BN / 2 : p.BN, false, kDenseHeader + table_bytes(slot_cp) + epi_bytes(false), 0).stages;
  p.row_tiles = 1;
  p.slot_boxes = slot_cp ? 0 : 1;
}

cudaError_t launch_dense16_dweight(const DWeightParams& r, int dtype, cudaStream_t st) {
  DenseParams p{};
  p.Rows = r.Xsrc; p.Slot = r.Ysrc; p.Ind = r.Ind; p.Out = r.out; p.acc = r.acc; p.status = r.status;
  p.B = r.B; p.T = r.T; p.E = r.E; p.K = r.K; p.M = r.M;
  p.swap = r.swap;
  p.C = r.swap ? r.FD : r.FG;
  p.N = r.swap ? r.FG : r.FD;
  p.lane_rows = (r.out_layout == EGS_DW_DIRECT_ROWS) == (r.swap != 0);
  p.index_dtype = r.index_dtype;
  p.BN = r.BN; p.stages = r.stages; p.splits = r.splits; p.rows_per_split = r.rows_per_split;
  p.half = r.pair ? r.BN / 2 : r.BN;
  p.after_own = r.after_own;
  const int rows = r.pair ? 2 * kTileM : kTileM;
  p.tiles_m = (p.C + rows - 1) / rows;
  p.tiles_n = (p.N + r.BN - 1) / r.BN;
  p.group = 1;
  p.full_waves = 0;
  p.groups_n = p.tiles_n;
  p.a_slots = p.stages;
  p.readers = kEpiWarps;
  p.r1 = Div(p.tiles_m);
  p.r2 = Div(p.splits);
  const long long units = static_cast<long long>(p.tiles_m) * p.tiles_n * p.E * p.splits;
  if (units > 2147483647ll - kSms) return cudaErrorInvalidValue;
  p.units = static_cast<int>(units);
  plan_walk(p, r.pair != 0);
  TensorMap3 mw{}, mr{};
  p.tma_rows = r.slot_boxes;
  if (p.tma_rows) {
    const int staged = r.swap ? kTileM : p.half;               // columns of the slot rows that a CTA stages
    p.whole = whole_segments(r.FD, staged, !r.swap && r.pair);
    p.boxes = p.whole ? 1 : (staged + 63) / 64;
    const unsigned long long kk = static_cast<unsigned long long>(r.K), fd = static_cast<unsigned long long>(r.FD), e = static_cast<unsigned long long>(r.E);
    const unsigned rows_k = static_cast<unsigned>(r.K < kStep ? r.K : kStep);
    const unsigned long long segs[5] = {p.whole ? 64ull : fd, kk, static_cast<unsigned long long>(r.B), p.whole ? fd / 64 : 1ull, e};
    const unsigned long long strides[4] = {fd * 2, e * kk * fd * 2, 128ull, kk * fd * 2};
    const unsigned seg_box[5] = {64u, rows_k, static_cast<unsigned>(kStep) / rows_k, p.whole ? static_cast<unsigned>(staged / 64) : 1u, 1u};
    if (!encode_tensor_map_16bit_strided(&mr, r.Ysrc, 5, segs, strides, seg_box)) return cudaErrorInvalidValue;
  }
  if (r.pair && (!encode_gather(&mw, r.Xsrc, static_cast<long long>(r.B) * r.T, r.FG) ||
                 (!p.tma_rows && !encode_gather(&mr, r.Ysrc, static_cast<long long>(r.M) * r.E, r.FD))))
    return cudaErrorInvalidValue;
  return r.pair ? launch_typed<kOpDweight, true>(p, dtype, mw, mr, st)
                : launch_typed<kOpDweight, false>(p, dtype, mw, mr, st);
}

}  // namespace egs

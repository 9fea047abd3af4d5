// Strict float32 on the tensor cores (sm_100a): operators G, S and D as one persistent, warp-specialised kernel.
//
// Every product is three TF32 products, lo*hi + hi*lo + hi*hi with hi = the top 19 bits of a float32 and lo = tf32(x - hi), so
// every operand exists twice.  The tensor core takes a TF32 operand from the top 19 bits of a word and ignores the rest: the raw
// float32 words ARE the hi operand, and a split pass only has to make the lo one.
//
//   warps 0..3    TMA gathers, four rows at a time (tile::gather4): token rows through Ind (G, D), slot rows that are no boxes
//   warps 4..15   splits, three groups of four warps that take the steps in turn.  The rows' operand goes from its raw tile through
//                 registers into tensor memory, hi and lo, and is the A operand of the MMAs (in D, whose contraction runs down the
//                 tile, a thread reads a column and the turn comes for free); of the columns' operand (weights; D: slot rows) the
//                 raw tile is the hi part, the lo part is written beside it
//   warps 16..23  read-out; where every step has an accumulator of its own they add those up in registers
//   then          one warp each for the MMAs, the TMA boxes, and the look-up of source and destination rows (D: contraction rows)
//
// What bounds it: the tensor core and shared memory, about equally.  A step multiplies 128 x BN by 32 contraction elements: at BN = 128
// twelve tcgen05.mma of 64 clocks each, 768.  The TMA writes 32 KB, the splits read 32 KB and write 16, the MMAs read 4 KB of their column
// operand each: 128 KB, 1000 clocks at 128 bytes a clock.  (With the rows' operand in shared memory too it was 192 KB, and with copies and
// splits in the same sixteen warps a step took 2150 clocks: the chain copy, wait, split, fence, multiply, free ran over two lo buffers.)
// A split takes 1400 clocks from its first wait to its arrival, hence three groups.  A step takes 1200-1300 clocks, with an accumulator
// per step 1600: eight warps then read and add 64 KB of tensor memory a step.
// 32768 routed rows, E = 32, I = 1024, J = 256, from cold caches: S 142 -> 99 us, D 173 -> 94, G 157 -> 127; 65536 rows, E = 32, I = 128,
// J = 64: 29 -> 23, 31 -> 23, 29 -> 23.
// The tensor core adds product groups into its accumulator with truncation, an error that grows with the number of steps
// (3.3e-5 of max|ref| at a contraction of 4096).  G and S up to a contraction of 512 and D, in ranges of at most 1024 rows, stay
// below 1.2e-5.  A longer contraction of G and S (LONG) takes an accumulator per step, the small products first, and sums the steps in
// registers of the read-out warps with correct rounding: 2.0e-7 to 2.6e-7 against float64 (2-norm, normal and positive values,
// 516 to 2048 elements), where FFMA sums have 3.5e-7 to 8.1e-7 and accumulators of 16, 4 and 2 steps 1.1e-5, 2.1e-6 and 8.2e-7.
// (Operands below 2^-110 lose their lo parts to the smallest exponent: 2e-5.)  The registers come from the producers (setmaxnreg).
#include "egs_tcgen05.cuh"

namespace egs {

namespace {

constexpr int kGatherWarps = 4, kSplitGroups = 3;
constexpr int kProdWarps = kGatherWarps + 4 * kSplitGroups;
// Read-out warps, each with half of a tile's columns (four warps took as long to add a scatter's tile as a contraction of 256 to multiply).
constexpr int kEpiWarps = 8;
constexpr int kMmaWarp = kProdWarps + kEpiWarps, kTmaWarp = kMmaWarp + 1, kIndexWarp = kMmaWarp + 2;
constexpr int kStrictThreads = (kIndexWarp + 2) * 32;
// Steps whose split operands exist, one per group.  Tensor memory (512 columns) holds their 64 columns each beside two accumulators.
constexpr int kOps = kSplitGroups, kAccs = 2;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kStrictHeader = 1024;
constexpr int kBatch = 128;                        // D: contraction rows whose ids are looked up at a time (four steps)
// G, S: source rows of two units, then destination rows of two units (-1: none).  D: token rows of two batches, then slot rows.
constexpr uint32_t kRowTable = 4u * kTileM * 4u;
static_assert(kBatch == kTileM, "one table serves both");
constexpr uint32_t kXpose = kEpiWarps * 4096u;      // transposes of the read-out
constexpr int kStepElems = 32;                     // contraction elements per step: one 128-byte segment of float32
constexpr uint32_t kSeg = kStepElems * 128u;       // 32 columns of a tile whose rows are contraction elements
constexpr int kWholeSteps = 16;                    // G / S: steps of a contraction that one accumulator sees whole (512 elements)
// Longer ones: registers a thread of the gathers and the last four warps, the splits, and the read-out; 28 warps of 72 at launch.
constexpr int kLongRestRegs = 40, kLongSplitRegs = 56, kLongEpiRegs = 128;
constexpr int kLongRegs = (kGatherWarps + 4) * kLongRestRegs + 4 * kSplitGroups * kLongSplitRegs + kEpiWarps * kLongEpiRegs;
static_assert(kLongRegs <= 28 * 72, "more registers than the block has");
constexpr uint32_t kATile = kTileM * 128u;         // bytes of a raw A tile; D: 32 rows of 128 features, the same
constexpr size_t kSmemMax = 227 * 1024;
constexpr int kSms = 148;

enum { kOpGather = 0, kOpScatter = 1, kOpDweight = 2 };

struct __align__(16) StrictHeader {
  unsigned long long a_full[kMaxStages];             // a raw tile has landed
  unsigned long long a_empty[kMaxStages];            // its group has read it
  unsigned long long b_full[kMaxStages];
  unsigned long long b_empty[kMaxStages];            // the step's MMAs are done: its raw B tile and its split operands may be overwritten
  unsigned long long split[kOps];                    // a step's split operands are ready
  unsigned long long acc_full[kAccs];
  unsigned long long acc_empty[kAccs];
  unsigned long long ids_full[2];
  unsigned long long ids_empty[2];
  unsigned long long dst_full[2];
  unsigned long long dst_empty[2];
  unsigned long long drain;
  uint32_t tmem_base;
  uint32_t abort_flag;
};
static_assert(sizeof(StrictHeader) <= kStrictHeader, "header does not fit");

struct StrictParams {
  const void* A;      // G, D: token rows; S: slot rows
  const void* Bsrc;   // G, S: weights; D: slot rows
  const void* bias;
  const void* Ind;
  float* Out;         // G: slot rows, S: token rows (added to), D: the weight gradient
  StatusRef status;
  int B, T, E, K, M;
  int C, N;           // G, S: contraction and produced width; D: C = FG (gathered features), N = FD
  int nc;             // G, S: 1 = weights [E, N, C]
  int index_dtype, out_layout;
  int BN;             // 32, 64, 96 or 128
  int raw_a, raw_b;   // raw tiles of A, of B
  int splits, rows_per_split;     // D
  int tiles_m, tiles_n;           // G, S: 128-row blocks per expert; D: 128-feature blocks; columns in BN
  int units;
  Div by_tiles_n, by_tiles_m, by_splits, stride, by_k;       // see Walk; stride: CTAs
  int step[4];                    // digits of the stride
  int slot_boxes;     // S, D: slot rows come as boxes
  int after_own;      // see launch_kernel
};

// The units of a CTA, a grid's width apart: column tile, row block, (D) row range, expert, the first fastest - the CTAs in flight share
// weights and rows in L2.  Advanced by adding the stride's digits, without divisions.
template <int OP>
struct Walk {
  int left;                       // units to come, this one included
  int e, m0, n0, split;
  int d0, d1, d2, d3;
  const StrictParams& p;
  __device__ __forceinline__ explicit Walk(const StrictParams& q) : p(q) {
    int u = blockIdx.x;
    left = u < p.units ? p.stride.quotient(p.units - u + p.stride.d - 1) : 0;
    d0 = p.by_tiles_n.remainder(u);
    d1 = p.by_tiles_m.remainder(u);
    d2 = OP == kOpDweight ? p.by_splits.remainder(u) : 0;
    d3 = u;
    place();
  }
  __device__ __forceinline__ void place() {
    n0 = d0 * p.BN;
    m0 = d1 * kTileM;
    split = d2;
    e = d3;
  }
  __device__ __forceinline__ void next() {
    --left;
    d0 += p.step[0];
    d1 += p.step[1];
    d2 += p.step[2];
    d3 += p.step[3];
    if (d0 >= p.tiles_n) { d0 -= p.tiles_n; ++d1; }
    if (d1 >= p.tiles_m) { d1 -= p.tiles_m; ++d2; }
    if (d2 >= (OP == kOpDweight ? p.splits : 1)) { d2 -= OP == kOpDweight ? p.splits : 1; ++d3; }
    place();
  }
  // contraction elements (D: rows) of the unit, and its steps
  __device__ __forceinline__ int length() const {
    return OP == kOpDweight ? min(p.rows_per_split, p.M - split * p.rows_per_split) : p.C;
  }
  __device__ __forceinline__ int steps() const { return (length() + kStepElems - 1) / kStepElems; }
};
// Position in a ring of raw tiles (of at least four).
struct Cursor {
  int slot = 0, round = 0;
  __device__ __forceinline__ void next(int stages, int by = 1) {
    slot += by;
    if (slot >= stages) {
      slot -= stages;
      ++round;
    }
  }
};

// lo = tf32(x - trunc19(x)), rounded to nearest (ties away) by adding half a unit of the last of the 19 bits; the bits below are left as
// they are, the tensor core ignores them
__device__ __forceinline__ uint32_t lo_part(uint32_t x) {
  const float rem = __uint_as_float(x) - __uint_as_float(x & 0xFFFFE000u);
  return __float_as_uint(rem) + 0x1000u;
}
__device__ __forceinline__ uint4 load_chunk(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok;
}
// tcgen05.mma (TF32) with the A operand in tensor memory: lane = row, a column per contraction element
__device__ __forceinline__ void umma_ts_tf32(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
      "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tma_gather4(uint32_t dst, const void* map, int x, const int (&r)[4], uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
      "l"(map), "r"(x), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const void* map, int x, int y, int z, int w, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void load_quad(uint32_t addr, int (&r)[4]) {
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

// Sums of a long contraction, two in a 64-bit register, each rounded to nearest.  (Held as single words they had to be paired and taken
// apart again at every addition: G 127 us against 132.)
__device__ __forceinline__ void add2(unsigned long long& sum, uint32_t x0, uint32_t x1) {
  asm("{\n\t.reg .b64 x;\n\tmov.b64 x, {%1, %2};\n\tadd.rn.f32x2 %0, %0, x;\n\t}" : "+l"(sum) : "r"(x0), "r"(x1));
}
__device__ __forceinline__ unsigned long long pair_of(uint32_t x0, uint32_t x1) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(x0), "r"(x1));
  return r;
}

// map_a: rows of A one by one (gather4) or as boxes; map_b: weights, or D's slot rows one by one or as boxes
template <int OP, bool LONG>
__global__ void __launch_bounds__(kStrictThreads, 1) strict_kernel(const __grid_constant__ StrictParams p, const __grid_constant__ TensorMap3 map_a,
                                                                         const __grid_constant__ TensorMap3 map_b) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  StrictHeader* hdr = reinterpret_cast<StrictHeader*>(smem_raw);
  const uint32_t smem0 = smem_u32(smem_raw);
  const uint32_t table = smem0 + kStrictHeader, xpose0 = table + kRowTable;
  const uint32_t b_bytes = static_cast<uint32_t>(p.BN) * 128u;
  const int raw_a = p.raw_a, raw_b = p.raw_b;
  const uint32_t a0 = xpose0 + kXpose, b0 = a0 + static_cast<uint32_t>(raw_a) * kATile, lo0 = b0 + static_cast<uint32_t>(raw_b) * b_bytes;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool gathers = OP != kOpScatter || !p.slot_boxes;
  volatile uint32_t* abort_flag = &hdr->abort_flag;

  if (tid == 0) {
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(smem_u32(&hdr->a_full[s]), 1);
      mbar_init(smem_u32(&hdr->a_empty[s]), 4);
      mbar_init(smem_u32(&hdr->b_full[s]), 1);
      mbar_init(smem_u32(&hdr->b_empty[s]), 1);
    }
    for (int o = 0; o < kOps; ++o) mbar_init(smem_u32(&hdr->split[o]), 4);
    for (int b = 0; b < kAccs; ++b) {
      mbar_init(smem_u32(&hdr->acc_full[b]), 1);
      mbar_init(smem_u32(&hdr->acc_empty[b]), kEpiWarps);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&hdr->ids_full[b]), OP == kOpDweight ? 64 : 32);
      mbar_init(smem_u32(&hdr->ids_empty[b]), kGatherWarps);
      mbar_init(smem_u32(&hdr->dst_full[b]), 32);
      mbar_init(smem_u32(&hdr->dst_empty[b]), kEpiWarps);
    }
    mbar_init(smem_u32(&hdr->drain), 1);
    fence_mbar_init();
    if (!p.after_own) pdl_wait();
    hdr->abort_flag = p.status.timed_out() ? 1u : 0u;
    if (smem_misaligned(smem_raw)) {
      hdr->abort_flag = 1u;
      p.status.report(EGS_STATUS_INTERNAL);
    }
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_u32(&hdr->tmem_base), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = hdr->tmem_base;
  const uint32_t acc_cols = tmem_cols_for(p.BN), ops_col = kAccs * acc_cols;     // accumulators, then per step 32 hi and 32 lo columns

  if (!p.after_own) pdl_wait();
  if (hdr->abort_flag != 0u) {
    pdl_wait();                                          // (and fall through to the common exit)
  } else if (warp < kProdWarps) {
    bool alive = true;
    if (warp < kGatherWarps) {
      if (LONG) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kLongRestRegs));
      // =========================== loads of A: gathers, four rows at a time, or slot rows in boxes ===========================
      Cursor at;
      auto take = [&]() {                                // the tile to load, once it is free
        if (at.round > 0) alive = mbar_wait_all(smem_u32(&hdr->a_empty[at.slot]), (at.round - 1) & 1, abort_flag, p.status.word);
        const int slot = at.slot;
        at.next(raw_a);
        return slot;
      };
      if (OP == kOpScatter && p.slot_boxes) {
        const int steps = (p.C + kStepElems - 1) / kStepElems;
        for (Walk<OP> u(p); warp == 0 && u.left > 0 && alive; u.next()) {
          const int b = p.by_k.quotient(u.m0), k = u.m0 - b * p.K;
          for (int ks = 0; ks < steps; ++ks) {
            const int slot = take();
            if (!alive) break;
            const uint32_t bar = smem_u32(&hdr->a_full[slot]);
            if (elect_one()) {
              mbar_arrive_expect_tx(bar, kATile);
              tma_load_4d(a0 + static_cast<uint32_t>(slot) * kATile, &map_a, ks * kStepElems, k, u.e, b, bar);
            }
          }
        }
      } else if constexpr (OP != kOpDweight) {
        constexpr int kQuads = kTileM / kGatherWarps / 4;
        const int steps = (p.C + kStepElems - 1) / kStepElems;
        int t = 0;
        for (Walk<OP> u(p); u.left > 0 && alive; u.next(), ++t) {
          alive = mbar_wait_all(smem_u32(&hdr->ids_full[t & 1]), (t >> 1) & 1, abort_flag, p.status.word);
          const uint32_t ids = table + static_cast<uint32_t>((t & 1) * kTileM + warp * kQuads * 4) * 4u;
          for (int k = 0; k < steps && alive; ++k) {
            const int slot = take();
            if (!alive) break;
            const uint32_t bar = smem_u32(&hdr->a_full[slot]);
            const uint32_t dst = a0 + static_cast<uint32_t>(slot) * kATile + static_cast<uint32_t>(warp * kQuads) * 512u;
            if (elect_one()) {
              if (warp == 0) mbar_arrive_expect_tx(bar, kATile);       // (for all four warps)
#pragma unroll
              for (int q0 = 0; q0 < kQuads; q0 += 4) {
                int row[4][4];
#pragma unroll
                for (int q = 0; q < 4; ++q) load_quad(ids + (q0 + q) * 16u, row[q]);
#pragma unroll
                for (int q = 0; q < 4; ++q) tma_gather4(dst + (q0 + q) * 512u, &map_a, k * kStepElems, row[q], bar);
              }
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&hdr->ids_empty[t & 1]));
        }
      } else {
        constexpr int kQuads = kStepElems / kGatherWarps / 4, kBatchSteps = kBatch / kStepElems;
        const int nseg = p.BN / 32;
        Cursor b_at;                                     // (slot rows that are no boxes come this way too)
        int batch = 0;
        for (Walk<OP> u(p); u.left > 0 && alive; u.next()) {
          const int steps = u.steps();
          for (int k = 0; k < steps; ++k) {
            const int in_batch = k % kBatchSteps;
            if (in_batch == 0) alive = mbar_wait_all(smem_u32(&hdr->ids_full[batch & 1]), (batch >> 1) & 1, abort_flag, p.status.word);
            if (!alive) break;
            int tok[kQuads][4], slot_row[kQuads][4];
            const uint32_t ids = table + static_cast<uint32_t>((batch & 1) * kBatch + in_batch * kStepElems + warp * kQuads * 4) * 4u;
#pragma unroll
            for (int q = 0; q < kQuads; ++q) {
              load_quad(ids + q * 16u, tok[q]);
              if (!p.slot_boxes) load_quad(ids + 2u * kBatch * 4u + q * 16u, slot_row[q]);
            }
            if (in_batch == kBatchSteps - 1 || k + 1 == steps) {                   // this warp has read the batch
              __syncwarp();
              if (lane == 0) mbar_arrive(smem_u32(&hdr->ids_empty[batch & 1]));
              ++batch;
            }
            const int slot = take();
            if (!alive) break;
            const uint32_t bar = smem_u32(&hdr->a_full[slot]);
            if (elect_one()) {
              if (warp == 0) mbar_arrive_expect_tx(bar, kATile);
#pragma unroll
              for (int q = 0; q < kQuads; ++q)           // (128 features a row)
                tma_gather4(a0 + static_cast<uint32_t>(slot) * kATile + static_cast<uint32_t>(warp * kQuads + q) * 2048u, &map_a, u.m0, tok[q], bar);
            }
            if (p.slot_boxes) continue;
            if (b_at.round > 0) alive = mbar_wait_all(smem_u32(&hdr->b_empty[b_at.slot]), (b_at.round - 1) & 1, abort_flag, p.status.word);
            if (!alive) break;
            const uint32_t b_bar = smem_u32(&hdr->b_full[b_at.slot]), b_dst = b0 + static_cast<uint32_t>(b_at.slot) * b_bytes;
            b_at.next(raw_b);
            if (elect_one()) {
              if (warp == 0) mbar_arrive_expect_tx(b_bar, b_bytes);
              for (int s = 0; s < nseg; ++s)
#pragma unroll
                for (int q = 0; q < kQuads; ++q)
                  tma_gather4(b_dst + s * kSeg + static_cast<uint32_t>(warp * kQuads + q) * 512u, &map_b, u.n0 + s * 32, slot_row[q], b_bar);
            }
          }
        }
      }
      __syncwarp();
    } else {
      // =========================== splits: every third step of the CTA ===========================
      if (LONG) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kLongSplitRegs));
      const int group = (warp - kGatherWarps) >> 2, row = (warp & 3) * 32 + lane;
      const uint32_t a_out = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + ops_col + static_cast<uint32_t>(group) * 64u;
      const uint32_t mine = static_cast<uint32_t>(row) * 16u, b_out = lo0 + static_cast<uint32_t>(group) * b_bytes + mine;
      constexpr uint32_t kPass = 128u * 16u;
      int total = 0;                                     // steps of this CTA
      if (OP != kOpDweight) total = Walk<OP>(p).left * ((p.C + kStepElems - 1) / kStepElems);
      else
        for (Walk<OP> u(p); u.left > 0; u.next()) total += u.steps();
      Cursor a_at, b_at, gone;                           // raw tiles of step g; step g - kOps, whose MMAs free this group's operands
      a_at.next(raw_a, group);
      b_at.next(raw_b, group);
      gone = b_at;
      // (the wait for step g - kOps stands before those for the tiles: this group does not see every phase of their barriers, and a
      // parity only tells a phase from its neighbour.  The MMAs of step g - kOps are done, so all tiles up to it have landed.)
      for (int g = group; g < total; g += kOps) {
        if (g >= kOps) {
          alive = mbar_wait_all(smem_u32(&hdr->b_empty[gone.slot]), gone.round & 1, abort_flag, p.status.word);
          if (!alive) break;
          gone.next(raw_b, kOps);
          tc_fence_after();
        }
        alive = mbar_wait_all(smem_u32(&hdr->a_full[a_at.slot]), a_at.round & 1, abort_flag, p.status.word);
        if (!alive) break;
        const uint32_t a_in = a0 + static_cast<uint32_t>(a_at.slot) * kATile, a_empty = smem_u32(&hdr->a_empty[a_at.slot]);
        a_at.next(raw_a, kOps);
#pragma unroll
        for (int h = 0; h < 2; ++h) {                    // a thread has a row, sixteen elements at a time
          uint32_t x[16], lo[16];
          if constexpr (OP != kOpDweight) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const uint4 v = load_chunk(a_in + static_cast<uint32_t>(row) * 128u + (static_cast<uint32_t>((h * 4 + c) ^ (row & 7)) << 4));
              x[4 * c] = v.x; x[4 * c + 1] = v.y; x[4 * c + 2] = v.z; x[4 * c + 3] = v.w;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              asm volatile("ld.shared.b32 %0, [%1];" : "=r"(x[i]) : "r"(a_in + static_cast<uint32_t>(h * 16 + i) * 512u + static_cast<uint32_t>(row) * 4u) : "memory");
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) lo[i] = lo_part(x[i]);
          tmem_st16(a_out + static_cast<uint32_t>(h) * 16u, x);
          tmem_st16(a_out + 32u + static_cast<uint32_t>(h) * 16u, lo);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(a_empty);
        alive = mbar_wait_all(smem_u32(&hdr->b_full[b_at.slot]), b_at.round & 1, abort_flag, p.status.word);
        if (!alive) break;
        const uint32_t b_in = b0 + static_cast<uint32_t>(b_at.slot) * b_bytes + mine;
        b_at.next(raw_b, kOps);
        // the lo tile has the raw tile's layout, so it is split chunk by chunk without looking at that
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint4 x[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if ((h * 4 + j) * kPass < b_bytes) x[j] = load_chunk(b_in + (h * 4 + j) * kPass);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if ((h * 4 + j) * kPass < b_bytes)
              asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(b_out + (h * 4 + j) * kPass), "r"(lo_part(x[j].x)), "r"(lo_part(x[j].y)),
                           "r"(lo_part(x[j].z)), "r"(lo_part(x[j].w))
                           : "memory");
        }
        fence_proxy_async_smem();
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&hdr->split[group]));
      }
    }
  } else if (warp < kMmaWarp) {
    // =========================== read-out ===========================
    if (LONG) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kLongEpiRegs));
    constexpr int kShares = kEpiWarps / 4, kBlocks = 4 / kShares;      // (the widest tile has four blocks of 32 columns)
    const int ew = warp - kProdWarps;
    const int lg = ew & 3, share = ew >> 2;              // TMEM lane group, share of the blocks
    const uint32_t tile = xpose0 + static_cast<uint32_t>(ew) * 4096u;
    const uint32_t lane_base = static_cast<uint32_t>(lg * 32) << 16;
    bool alive = true;
    pdl_wait();                                          // the zeros the results are added to
    int buf = 0, around = 0;                             // next accumulator, times through all of them
    int t = 0;
    for (Walk<OP> u(p); u.left > 0 && alive; u.next(), ++t) {
      const int steps = u.steps();
      int my_ro = -1;                                    // G, S: destination row of tile row lg * 32 + lane
      if (OP != kOpDweight) {
        alive = mbar_wait_all(smem_u32(&hdr->dst_full[t & 1]), (t >> 1) & 1, abort_flag, p.status.word);
        if (!alive) break;
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(my_ro) : "r"(table + static_cast<uint32_t>((2 + (t & 1)) * kTileM + lg * 32 + lane) * 4u) : "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&hdr->dst_empty[t & 1]));
      }
      const int bn = min(p.BN, p.N - u.n0);
      const int nblk = (bn + 31) >> 5;
      auto wait_full = [&]() {
        alive = mbar_wait_all(smem_u32(&hdr->acc_full[buf]), around & 1, abort_flag, p.status.word);
        if (alive) tc_fence_after();
        return tmem_base + lane_base + static_cast<uint32_t>(buf) * acc_cols;
      };
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&hdr->acc_empty[buf]));
        if (++buf == kAccs) { buf = 0; ++around; }
      };
      auto emit = [&](int c, const uint32_t (&w)[32]) {
          const int col0 = u.n0 + c * 32;
          if (OP != kOpDweight) {
            warp_regs_emit(w, tile, lane, [&](int row, int cj, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3) {
              const int ro = __shfl_sync(0xffffffffu, my_ro, row);
              const int col = col0 + cj;
              if (ro >= 0 && col < p.N) {
                if (p.bias) add_bias4<float>(static_cast<const float*>(p.bias) + static_cast<long long>(u.e) * p.N + col, x0, x1, x2, x3);
                float* out = p.Out + static_cast<long long>(ro) * p.N + col;
                if (OP == kOpScatter) red4(out, x0, x1, x2, x3);
                else store4(out, x0, x1, x2, x3);
              }
            });
          } else if (p.out_layout == EGS_DW_GATHERED_ROWS) {     // out[e, f, g]: rows f are contiguous over g
            warp_regs_emit(w, tile, lane, [&](int row, int cj, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3) {
              const int f = u.m0 + lg * 32 + row, g = col0 + cj;
              if (f < p.C && g < p.N) {
                float* out = p.Out + (static_cast<long long>(u.e) * p.C + f) * p.N + g;
                if (p.splits > 1) red4(out, x0, x1, x2, x3);
                else store4(out, x0, x1, x2, x3);
              }
            });
          } else {                                               // out[e, g, f]: lanes f are contiguous for a fixed g
            const int f = u.m0 + lg * 32 + lane;
            if (f < p.C) {
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                if (col0 + i < p.N) {
                  float* out = p.Out + (static_cast<long long>(u.e) * p.N + col0 + i) * p.C + f;
                  if (p.splits > 1) atomicAdd(out, __uint_as_float(w[i]));
                  else *out = __uint_as_float(w[i]);
                }
              }
            }
          }
      };
      // An infinite operand times a zero lo part is NaN where the float32 product is infinite: sums that came out as NaN are formed
      // again, one product after the other as the generic kernel does.
      auto again_if_nan = [&](int c, uint32_t (&w)[32]) {
        bool nan = false;
#pragma unroll
        for (int i = 0; i < 32; ++i) nan |= isnan(__uint_as_float(w[i]));
        if (!__any_sync(0xffffffffu, nan)) return;
        const int m = u.m0 + lg * 32 + lane, b = m / p.K, slot = (b * p.E + u.e) * p.K + (m - b * p.K);
        int row = m < p.M ? slot : -1;
        if (OP == kOpGather && row >= 0) {
          const long long tk = load_index(p.Ind, p.index_dtype, slot);
          row = tk >= 0 && tk < p.T ? b * p.T + static_cast<int>(tk) : -1;
        }
        const float* a = static_cast<const float*>(p.A) + static_cast<long long>(row) * p.C;
        const float* wt = static_cast<const float*>(p.Bsrc) + static_cast<long long>(u.e) * p.C * p.N;
#pragma unroll
        for (int i = 0; i < 32; ++i) asm volatile("st.shared.b32 [%0], %1;" ::"r"(tile + i * 128u + lane * 4u), "r"(w[i]) : "memory");
#pragma unroll 1
        for (int i = 0; i < 32; ++i) {
          float x;
          const int n = u.n0 + c * 32 + i;
          asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(tile + i * 128u + lane * 4u) : "memory");
          if (m < p.M && n < p.N && isnan(x)) {
            x = 0.f;
#pragma unroll 1
            for (int k = 0; k < p.C; ++k)
              x = fmaf(row >= 0 ? a[k] : 0.f, wt[p.nc ? static_cast<long long>(n) * p.C + k : static_cast<long long>(k) * p.N + n], x);
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(tile + i * 128u + lane * 4u), "f"(x) : "memory");
          }
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w[i]) : "r"(tile + i * 128u + lane * 4u) : "memory");
        __syncwarp();
      };
      if (LONG) {
        unsigned long long v[kBlocks][16];               // the sums of this thread's row, in pairs
        for (int ch = 0; ch < steps; ++ch) {
          const uint32_t acc = wait_full();
          if (!alive) break;
#pragma unroll
          for (int c = 0; c < kBlocks; ++c) {
            if (c * kShares + share < nblk) {
              uint32_t x[32];
              tmem_ld32(acc + static_cast<uint32_t>((c * kShares + share) * 32), x);
              tmem_ld_wait();
              if (ch == 0) {
#pragma unroll
                for (int i = 0; i < 16; ++i) v[c][i] = pair_of(x[2 * i], x[2 * i + 1]);
              } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) add2(v[c][i], x[2 * i], x[2 * i + 1]);
              }
            }
          }
          release();
        }
        if (!alive) break;
#pragma unroll
        for (int c = 0; c < kBlocks; ++c) {
          if (c * kShares + share < nblk) {
            uint32_t w[32];
#pragma unroll
            for (int i = 0; i < 16; ++i) asm("mov.b64 {%0, %1}, %2;" : "=r"(w[2 * i]), "=r"(w[2 * i + 1]) : "l"(v[c][i]));
            again_if_nan(c * kShares + share, w);
            emit(c * kShares + share, w);
          }
        }
      } else {
        const uint32_t acc = wait_full();
        if (!alive) break;
        for (int c = share; c < nblk; c += kShares) {
          uint32_t v[32];
          tmem_ld32(acc + static_cast<uint32_t>(c * 32), v);
          tmem_ld_wait();
          emit(c, v);
        }
        release();
      }
    }
  } else {
    if (LONG) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kLongRestRegs));
    if (warp == kMmaWarp) {
      // =========================== MMA issuer ===========================
      // (the warp runs converged and an elected lane issues, see mbar_wait_all: twelve MMAs from a lane on its own took 1000 clocks)
      // B: rows = n (weights [n][contraction]) or rows = contraction
      const bool b_mn = OP == kOpDweight || !p.nc;
      const uint32_t b_lbo = b_mn ? kSeg : 16u, b_sbo = b_mn ? 512u : 1024u, b_lay = b_mn ? kSwizzle128Base32 : kSwizzle128;
      const uint32_t b_adv = (b_mn ? 8u * 128u : 32u) >> 4;
      const uint64_t b_desc = make_smem_desc(0u, b_lbo, b_sbo, b_lay);
      // What the next step waits for is asked for between the MMAs of this one: a satisfied wait takes 150 clocks, and behind the last
      // MMA of a step the tensor core would run dry meanwhile (its queue holds a few of the twelve, which take 64 clocks each).
      auto seen = [&](uint32_t bar, int phase) { return __all_sync(0xffffffffu, mbar_test(bar, phase & 1) != 0u) != 0; };
      bool ok = true, split_seen = false, acc_seen = false;
      int buf = 0, around = 0, op = 0, op_round = 0;
      Cursor at;
      for (Walk<OP> u(p); u.left > 0 && ok; u.next()) {
        const int steps = u.steps(), len = u.length();
        const int bn = min(p.BN, ((p.N - u.n0) + 15) & ~15);
        const uint32_t idesc = make_idesc(2u, 0u, b_mn ? 1u : 0u, kTileM, static_cast<uint32_t>(bn));
        for (int ks = 0; ks < steps && ok; ++ks) {
          const bool first = LONG || ks == 0, last = LONG || ks == steps - 1;
          if (first && around > 0 && !acc_seen) {
            ok = mbar_wait_all(smem_u32(&hdr->acc_empty[buf]), (around - 1) & 1, abort_flag, p.status.word);
            if (!ok) break;
          }
          if (!split_seen) {
            ok = mbar_wait_all(smem_u32(&hdr->split[op]), op_round & 1, abort_flag, p.status.word);
            if (!ok) break;
          }
          tc_fence_after();
          const uint32_t d = tmem_base + static_cast<uint32_t>(buf) * acc_cols;
          // (descriptors: 14 address bits in 16-byte units; shared memory is smaller)
          const uint64_t b_hi = b_desc + ((b0 + static_cast<uint32_t>(at.slot) * b_bytes) >> 4);
          const uint64_t b_lo = b_desc + ((lo0 + static_cast<uint32_t>(op) * b_bytes) >> 4);
          const uint32_t a_hi = tmem_base + ops_col + static_cast<uint32_t>(op) * 64u, a_lo = a_hi + 32u;
          const int nkq = min(4, (len - ks * kStepElems + 7) / 8);
          const uint32_t empty = smem_u32(&hdr->b_empty[at.slot]);
          at.next(raw_b);
          auto hi_hi = [&](int kq) { umma_ts_tf32(d, a_hi + kq * 8, b_hi + kq * b_adv, idesc, 1u); };
          auto quarter = [&](int kq) {
            if (kq >= nkq) return;
            umma_ts_tf32(d, a_lo + kq * 8, b_hi + kq * b_adv, idesc, (first && kq == 0) ? 0u : 1u);
            umma_ts_tf32(d, a_hi + kq * 8, b_lo + kq * b_adv, idesc, 1u);
            if (!LONG) hi_hi(kq);
          };
          if (elect_one()) {
            quarter(0);
            quarter(1);
            if (LONG) {
              quarter(2);
              quarter(3);
            }
          }
          const uint32_t full = smem_u32(&hdr->acc_full[buf]);
          if (last && ++buf == kAccs) { buf = 0; ++around; }
          if (++op == kOps) { op = 0; ++op_round; }
          acc_seen = last && around > 0 && seen(smem_u32(&hdr->acc_empty[buf]), around - 1);
          split_seen = seen(smem_u32(&hdr->split[op]), op_round);
          if (elect_one()) {
            if (!LONG) {
              quarter(2);
              quarter(3);
            } else {                                     // the small products first: additions truncate, and to a small sum that is little
#pragma unroll
              for (int kq = 0; kq < 4; ++kq)
                if (kq < nkq) hi_hi(kq);
            }
            umma_commit(empty);
            if (last) umma_commit(full);
          }
        }
      }
      pdl_trigger();                                     // (not before: a dependent's waiting CTAs would keep a kernel of another stream off this SM)
    } else if (warp == kTmaWarp) {
      // =========================== loads of B in boxes ===========================
      const int nseg = p.BN / 32;
      bool ok = true;
      Cursor at;
      for (Walk<OP> u(p); (OP != kOpDweight || p.slot_boxes) && u.left > 0 && ok; u.next()) {
        const int steps = u.steps();
        const int m = OP == kOpDweight ? u.split * p.rows_per_split : 0;
        int b = p.by_k.quotient(m), k = m - b * p.K;     // D: first slot row of the step
        for (int ks = 0, c0 = 0; ks < steps; ++ks, c0 += kStepElems) {
          if (at.round > 0) ok = mbar_wait_all(smem_u32(&hdr->b_empty[at.slot]), (at.round - 1) & 1, abort_flag, p.status.word);
          if (!ok) break;
          const uint32_t bar = smem_u32(&hdr->b_full[at.slot]), base = b0 + static_cast<uint32_t>(at.slot) * b_bytes;
          at.next(raw_b);
          if (elect_one()) {
            mbar_arrive_expect_tx(bar, b_bytes);
            if (OP != kOpDweight && p.nc) {
              tma_load_3d(base, &map_b, c0, u.n0, u.e, bar);
            } else {
              for (int s = 0; s < nseg; ++s) {
                if (OP != kOpDweight) tma_load_3d(base + s * kSeg, &map_b, u.n0 + s * 32, c0, u.e, bar);
                else tma_load_4d(base + s * kSeg, &map_b, u.n0 + s * 32, k, u.e, b, bar);
              }
            }
          }
          if (OP == kOpDweight) {
            k += kStepElems;                             // 32 rows are parts of one batch element or whole ones
            while (k >= p.K) { k -= p.K; ++b; }
          }
        }
      }
    } else {
      // =========================== index warps ===========================
      bool alive = true;
      if constexpr (OP != kOpDweight) {
        // the first warp: where the rows are; the second: where the read-out puts them
        const bool dst = warp != kIndexWarp;
        unsigned long long* full = dst ? hdr->dst_full : hdr->ids_full;
        unsigned long long* empty = dst ? hdr->dst_empty : hdr->ids_empty;
        int t = 0;
        for (Walk<OP> u(p); (dst || gathers) && u.left > 0 && alive; u.next(), ++t) {
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
        const int it = tid - kIndexWarp * 32;
        int batch = 0;
        for (Walk<OP> u(p); u.left > 0 && alive; u.next()) {
          const int m_begin = u.split * p.rows_per_split, m_end = m_begin + u.length();
          const bool report = u.m0 == 0 && u.n0 == 0;
          for (int m0 = m_begin; m0 < m_end && alive; m0 += kBatch, ++batch) {
            int tok[2], slot_row[2];
            long long t[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {                // both loads first
              const int m = m0 + it + i * 64;
              const bool on = m < m_end;
              tok[i] = on ? p.by_k.quotient(m) : 0;
              const int s = (tok[i] * p.E + u.e) * p.K + (on ? m - tok[i] * p.K : 0);
              t[i] = load_index(p.Ind, p.index_dtype, s);
              slot_row[i] = on ? s : -1;
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const bool known = t[i] >= 0 && t[i] < p.T;
              if (slot_row[i] >= 0 && !known && report) p.status.report(EGS_STATUS_INDEX_OUT_OF_RANGE);
              tok[i] = (slot_row[i] >= 0 && known) ? tok[i] * p.T + static_cast<int>(t[i]) : -1;
            }
            if (batch >= 2) alive = mbar_wait_all(smem_u32(&hdr->ids_empty[batch & 1]), ((batch >> 1) - 1) & 1, abort_flag, p.status.word);
            if (!alive) break;
            const uint32_t dst = table + static_cast<uint32_t>((batch & 1) * kBatch + it) * 4u;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + i * 256u), "r"(tok[i]) : "memory");
              if (!p.slot_boxes) asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + 2u * kBatch * 4u + i * 256u), "r"(slot_row[i]) : "memory");
            }
            mbar_arrive(smem_u32(&hdr->ids_full[batch & 1]));
          }
        }
      }
    }
    __syncwarp();
  }

  // ---- common exit ----
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) tmem_release(tmem_base, kTmemCols, smem_u32(&hdr->drain), abort_flag, p.status, lane);
}

// Tile width over n columns: what all tiles of a row block move through shared memory, n_tiles * (128 + BN) rows, decides.
int strict_bn(int n) {
  int best = 128, best_cost = 1 << 30;
  for (int bn = 32; bn <= 128; bn += 32) {
    const int cost = (n + bn - 1) / bn * (kTileM + bn);
    if (cost <= best_cost) {
      best = bn;
      best_cost = cost;
    }
  }
  return best;
}
bool long_contraction(int c) { return c > kWholeSteps * kStepElems; }
size_t strict_smem(int bn, int raw_a, int raw_b) {
  return kStrictHeader + kRowTable + kXpose + static_cast<size_t>(raw_a) * kATile + static_cast<size_t>(raw_b + kOps) * bn * 128;
}
// Raw tiles of B, which stay until they are multiplied, and of A, which are read one step and more before that: up to one less.
int strict_raw_b(int bn) {
  int raw = kMaxStages;
  while (strict_smem(bn, raw > 5 ? raw - 1 : 4, raw) > kSmemMax) --raw;
  return raw;
}
int strict_raw_a(int bn, int raw_b) { return strict_smem(bn, raw_b, raw_b) <= kSmemMax ? raw_b : raw_b > 5 ? raw_b - 1 : 4; }
// Slot rows can come as one TMA box where `rows` consecutive expert rows starting at a multiple of `rows` are whole batch elements or
// lie inside one.
bool rows_fit_boxes(int K, int rows) { return K % rows == 0 || rows % K == 0; }
bool encode_slot_boxes(TensorMap3* map, const void* base, int B, int E, int K, int width, int rows, bool mn) {
  const unsigned kk = static_cast<unsigned>(K < rows ? K : rows);
  const unsigned long long dims[4] = {static_cast<unsigned long long>(width), static_cast<unsigned long long>(K),
                                      static_cast<unsigned long long>(E), static_cast<unsigned long long>(B)};
  const unsigned box[4] = {32u, kk, 1u, static_cast<unsigned>(rows) / kk};
  return encode_tensor_map_32bit(map, base, 4, dims, box, mn ? kMapSwizzle128Base32 : kMapSwizzle128);
}
// rows one by one for tile::gather4, `cols` features at a time
bool encode_rows(TensorMap3* map, const void* base, long long rows, int width, int cols, int swizzle) {
  const unsigned long long dims[2] = {static_cast<unsigned long long>(width), static_cast<unsigned long long>(rows > 0 ? rows : 1)};
  const unsigned box[2] = {static_cast<unsigned>(cols), 1u};
  return encode_tensor_map_32bit(map, base, 2, dims, box, swizzle);
}

void plan_walk(StrictParams& p) {
  p.by_tiles_n = Div(p.tiles_n);
  p.by_tiles_m = Div(p.tiles_m);
  p.by_splits = Div(p.splits > 0 ? p.splits : 1);
  p.by_k = Div(p.K);
  p.stride = Div(p.units < kSms ? p.units : kSms);
  int s = p.stride.d;
  p.step[0] = s % p.tiles_n; s /= p.tiles_n;
  p.step[1] = s % p.tiles_m; s /= p.tiles_m;
  p.step[2] = s % p.by_splits.d;
  p.step[3] = s / p.by_splits.d;
}

template <int OP, bool LONG = false>
cudaError_t launch(const StrictParams& p, const TensorMap3& ma, const TensorMap3& mb, cudaStream_t st) {
  const size_t smem = strict_smem(p.BN, p.raw_a, p.raw_b);
  cudaError_t err = ensure_smem_optin<strict_kernel<OP, LONG>>(static_cast<int>(kSmemMax));
  if (err != cudaSuccess) return err;
  if (LONG) {                                            // setmaxnreg can only share out what the block is launched with
    static const int regs = [] {
      cudaFuncAttributes a{};
      return cudaFuncGetAttributes(&a, strict_kernel<OP, LONG>) == cudaSuccess ? a.numRegs : 0;
    }();
    if (regs * kStrictThreads < kLongRegs * 32) return cudaErrorInvalidConfiguration;
  }
  err = launch_kernel(strict_kernel<OP, LONG>, p.stride.d, kStrictThreads, smem, st, true, p, ma, mb);
  count_launch();
  return err;
}

}  // namespace

void configure_strict_rowgemm(RowGemmParams& p, bool scatter) {
  p.BN = strict_bn(p.N);
  p.slot_boxes = scatter && rows_fit_boxes(p.K, kTileM) ? 1 : 0;
  p.stages = strict_raw_b(p.BN);
  p.row_tiles = 1;
  p.persistent = 1;
}

cudaError_t launch_strict_rowgemm(const RowGemmParams& r, bool scatter, cudaStream_t st) {
  StrictParams p{};
  p.A = r.A; p.Bsrc = r.W; p.bias = r.bias; p.Ind = r.Ind; p.Out = static_cast<float*>(r.Out); p.status = r.status;
  p.B = r.B; p.T = r.T; p.E = r.E; p.K = r.K; p.M = r.M; p.C = r.C; p.N = r.N;
  p.nc = r.w_layout == EGS_W_NC;
  p.index_dtype = r.index_dtype;
  p.BN = r.BN; p.raw_b = r.stages; p.raw_a = strict_raw_a(r.BN, r.stages);
  p.after_own = r.after_own;
  p.tiles_m = (r.M + kTileM - 1) / kTileM;
  p.tiles_n = (r.N + r.BN - 1) / r.BN;
  const long long units = static_cast<long long>(p.tiles_m) * p.tiles_n * p.E;
  if (units > 2147483647ll) return cudaErrorInvalidValue;
  p.units = static_cast<int>(units);
  plan_walk(p);
  p.slot_boxes = r.slot_boxes;
  TensorMap3 ma{}, mb{};
  const unsigned long long inner = p.nc ? r.C : r.N, outer = p.nc ? r.N : r.C;
  const unsigned long long dims[3] = {inner, outer, static_cast<unsigned long long>(r.E)};
  const unsigned box[3] = {32u, p.nc ? static_cast<unsigned>(p.BN) : static_cast<unsigned>(kStepElems), 1u};
  if (!encode_tensor_map_32bit(&mb, r.W, 3, dims, box, p.nc ? kMapSwizzle128 : kMapSwizzle128Base32)) return cudaErrorInvalidValue;
  const bool a_ok = p.slot_boxes ? encode_slot_boxes(&ma, r.A, r.B, r.E, r.K, r.C, kTileM, false)
                                 : encode_rows(&ma, r.A, scatter ? static_cast<long long>(r.M) * r.E : static_cast<long long>(r.B) * r.T, r.C, 32, kMapSwizzle128);
  if (!a_ok) return cudaErrorInvalidValue;
  if (long_contraction(r.C))
    return scatter ? launch<kOpScatter, true>(p, ma, mb, st) : launch<kOpGather, true>(p, ma, mb, st);
  return scatter ? launch<kOpScatter>(p, ma, mb, st) : launch<kOpGather>(p, ma, mb, st);
}

void configure_strict_dweight(DWeightParams& p) {
  p.BN = strict_bn(p.FD);
  p.slot_boxes = rows_fit_boxes(p.K, kStepElems) ? 1 : 0;
  p.stages = strict_raw_b(p.BN);
  p.row_tiles = 1;
  // row ranges: as many as still leave one unit per SM, at most 1024 rows each (see the top of the file)
  const long long tiles = static_cast<long long>((p.FG + kTileM - 1) / kTileM) * ((p.FD + p.BN - 1) / p.BN) * p.E;
  long long want = kSms / tiles;
  const long long least = (p.M + 1023) / 1024, most = (p.M + kStepElems - 1) / kStepElems;
  if (want < least) want = least;
  if (want > most) want = most;
  if (want < 1) want = 1;
  long long rows = (p.M + want - 1) / want;
  rows = (rows + kStepElems - 1) / kStepElems * kStepElems;
  p.rows_per_split = static_cast<int>(rows);
  p.splits = static_cast<int>((p.M + rows - 1) / rows);
}

cudaError_t launch_strict_dweight(const DWeightParams& r, cudaStream_t st) {
  StrictParams p{};
  p.A = r.Xsrc; p.Bsrc = r.Ysrc; p.Ind = r.Ind; p.Out = static_cast<float*>(r.splits > 1 ? r.acc : r.out); p.status = r.status;
  p.B = r.B; p.T = r.T; p.E = r.E; p.K = r.K; p.M = r.M; p.C = r.FG; p.N = r.FD;
  p.index_dtype = r.index_dtype; p.out_layout = r.out_layout;
  p.BN = r.BN; p.raw_b = r.stages; p.raw_a = strict_raw_a(r.BN, r.stages);
  p.after_own = r.after_own;
  p.splits = r.splits; p.rows_per_split = r.rows_per_split;
  p.tiles_m = (r.FG + kTileM - 1) / kTileM;
  p.tiles_n = (r.FD + r.BN - 1) / r.BN;
  const long long units = static_cast<long long>(p.tiles_m) * p.tiles_n * p.E * p.splits;
  if (units > 2147483647ll) return cudaErrorInvalidValue;
  p.units = static_cast<int>(units);
  plan_walk(p);
  p.slot_boxes = r.slot_boxes;
  TensorMap3 ma{}, mb{};
  if (!encode_rows(&ma, r.Xsrc, static_cast<long long>(r.B) * r.T, r.FG, kTileM, kMapSwizzleNone) ||
      !(p.slot_boxes ? encode_slot_boxes(&mb, r.Ysrc, r.B, r.E, r.K, r.FD, kStepElems, true)
                     : encode_rows(&mb, r.Ysrc, static_cast<long long>(r.M) * r.E, r.FD, 32, kMapSwizzle128Base32)))
    return cudaErrorInvalidValue;
  return launch<kOpDweight>(p, ma, mb, st);
}

}  // namespace egs

// Strict float32 on the tensor cores (sm_100a): operators G, S and D as one persistent, warp-specialised kernel.
//
// Every product is three TF32 products, lo*hi + hi*lo + hi*hi with hi = the top 19 bits of a float32 and lo = tf32(x - hi), so
// every operand tile exists twice in shared memory.  The tensor core takes a TF32 operand from the top 19 bits of a word and
// ignores the rest: the raw float32 tile IS the hi tile, and only the lo tile is written by the split pass.
//
// What bounds it is shared-memory bandwidth.  A step multiplies 128 x BN by 32 contraction elements: the copies write
// (128 + BN) * 128 bytes, the split reads them and writes as much again, and the twelve tcgen05.mma read both operands three
// times over - at BN = 128 192 KB or 1500 clocks at 128 bytes per clock, against 768 clocks of tensor work.  Wide tiles
// therefore pay (at BN = 64 the same bytes serve half the products), and the rest is keeping those clocks busy:
//   * two rings.  Raw tiles are prefetched `raw - lo` steps ahead (each thread splits exactly the chunks it has copied itself, so
//     its own copy group is all it waits for); lo tiles need two buffers, the one the tensor core reads and the one being
//     written.  (One ring of hi+lo stages has room for two stages and therefore no prefetch: 1.9 us a step, most of it load latency.)
//   * persistent CTAs, the rings run on across tiles, the accumulator is double-buffered in tensor memory, and dedicated warps
//     read it out while the next tile is multiplied.
// The tensor core adds product groups into its accumulator with truncation, an error that grows with the number of steps
// (3.3e-5 of max|ref| at a contraction of 4096).  G and S up to a contraction of 512 and D, in ranges of at most 1024 rows, stay
// below 1.2e-5.  A longer contraction of G and S (LONG) takes an accumulator per step, the small products first, and sums the steps in
// registers of the read-out warps with correct rounding: 2.0e-7 to 2.6e-7 against float64 (2-norm, normal and positive values,
// 516 to 2048 elements), where FFMA sums have 3.5e-7 to 8.1e-7 and accumulators of 16, 4 and 2 steps 1.1e-5, 2.1e-6 and 8.2e-7.
// (Operands below 2^-110 lose their lo parts to the smallest exponent: 2e-5.)  The registers come from the producers (setmaxnreg).
// 32768 routed rows, I = 1024, J = 256: S 138 us, D 171, G 154 (FFMA 474).
#include "egs_tcgen05.cuh"

namespace egs {

namespace {

// Sixteen producer warps: a step costs a producer thread about 120 instructions for its (up to) four chunks, and with eight warps
// (two per scheduler) their latencies, not the shared-memory clocks, set the pace: 1.4 us per step instead of 1.1.
constexpr int kProdWarps = 16, kProdThreads = kProdWarps * 32;
// Read-out warps; twice as many, each with half of the columns, where they also add up a long contraction.
__host__ __device__ constexpr int epi_warps(bool long_c) { return long_c ? 8 : 4; }
// (long contractions: the register split is by warpgroups, see kLongProdRegs)
__host__ __device__ constexpr int strict_threads(bool long_c) { return (kProdWarps + epi_warps(long_c) + (long_c ? 4 : 1)) * 32; }
constexpr int kLoStages = 2;
constexpr uint32_t kStrictHeader = 1024;
__host__ __device__ constexpr uint32_t xpose_bytes(bool long_c) { return epi_warps(long_c) * 4096u; }
constexpr int kStepElems = 32;                     // contraction elements per step: one 128-byte segment of float32
constexpr int kWholeSteps = 16;                    // G / S: steps of a contraction that one accumulator sees whole (512 elements)
// Longer ones: registers a thread of the producers, the read-out and the MMA warp's group; 28 warps of 72 at launch.
constexpr int kLongProdRegs = 48, kLongEpiRegs = 144, kLongMmaRegs = 24;
static_assert(kProdWarps * kLongProdRegs + epi_warps(true) * kLongEpiRegs + 4 * kLongMmaRegs <= 28 * 72, "more registers than the block has");
constexpr uint32_t kATile = kTileM * 128u;         // bytes of a raw A tile; D: 32 rows of 128 features, the same
constexpr size_t kSmemMax = 227 * 1024;
constexpr int kSms = 148;

enum { kOpGather = 0, kOpScatter = 1, kOpDweight = 2 };

struct __align__(16) StrictHeader {
  unsigned long long full[kMaxStages];
  unsigned long long empty[kMaxStages];
  unsigned long long acc_full[4];
  unsigned long long acc_empty[4];
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
  int raw;            // raw stages
  int splits, rows_per_split;     // D
  int tiles_m, tiles_n;           // G, S: 128-row blocks per expert; D: 128-feature blocks; columns in BN
  int units;
  int after_own;      // see launch_kernel
};

struct Unit {
  int e, m0, n0, split;
};
// Units of one expert follow each other, the N tiles of one row block fastest: the CTAs in flight share weights and rows in L2.
template <int OP>
__device__ __forceinline__ Unit unit_of(const StrictParams& p, int u) {
  Unit r;
  const int nt = u % p.tiles_n;
  u /= p.tiles_n;
  const int mt = u % p.tiles_m;
  u /= p.tiles_m;
  r.split = 0;
  if (OP == kOpDweight) {
    r.split = u % p.splits;
    u /= p.splits;
  }
  r.e = u;
  r.m0 = mt * kTileM;
  r.n0 = nt * p.BN;
  return r;
}
// steps of a unit's contraction
template <int OP>
__device__ __forceinline__ int unit_steps(const StrictParams& p, const Unit& u) {
  if (OP != kOpDweight) return (p.C + kStepElems - 1) / kStepElems;
  const int rows = min(p.rows_per_split, p.M - u.split * p.rows_per_split);
  return (rows + kStepElems - 1) / kStepElems;
}

// lo = tf32(x - trunc19(x)) of the four words of a chunk, rounded to nearest (ties away) by adding half a unit of the last of the
// 19 bits; the bits below are left as they are, the tensor core ignores them
__device__ __forceinline__ void store_lo(uint32_t dst, const uint4& x) {
  const uint32_t v[4] = {x.x, x.y, x.z, x.w};
  uint32_t lo[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float rem = __uint_as_float(v[i]) - __uint_as_float(v[i] & 0xFFFFE000u);
    lo[i] = __float_as_uint(rem) + 0x1000u;
  }
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(lo[0]), "r"(lo[1]), "r"(lo[2]), "r"(lo[3]) : "memory");
}
__device__ __forceinline__ uint4 load_chunk(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t swz16(int c, int r) { return static_cast<uint32_t>((c & 7) ^ (r & 7)) << 4; }
__device__ __forceinline__ uint32_t swz32(int c, int r) {
  return (static_cast<uint32_t>(((c & 7) >> 1) ^ (r & 3)) << 5) + (static_cast<uint32_t>(c & 1) << 4);
}

__device__ __forceinline__ void add2(uint32_t& a0, uint32_t& a1, uint32_t b0, uint32_t b1) {
  asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %3};\n\tadd.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a;\n\t}"
      : "+r"(a0), "+r"(a1)
      : "r"(b0), "r"(b1));
}

template <int OP, bool LONG>
__global__ void __launch_bounds__(strict_threads(LONG), 1) strict_kernel(StrictParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  StrictHeader* hdr = reinterpret_cast<StrictHeader*>(smem_raw);
  const uint32_t smem0 = smem_u32(smem_raw);
  const uint32_t xpose0 = smem0 + kStrictHeader;
  constexpr int kEpiWarps = epi_warps(LONG), kMmaWarp = kProdWarps + kEpiWarps;
  constexpr int kAccs = LONG ? 4 : 2;                 // accumulators in tensor memory
  const uint32_t raw0 = xpose0 + xpose_bytes(LONG);
  const uint32_t stage_bytes = kATile + static_cast<uint32_t>(p.BN) * 128u;      // A then B, the same in the lo ring
  const uint32_t lo0 = raw0 + static_cast<uint32_t>(p.raw) * stage_bytes;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int raw = p.raw;
  const uint32_t acc_cols = tmem_cols_for(p.BN);
  const uint32_t tmem_cols = kAccs * acc_cols;
  volatile uint32_t* abort_flag = &hdr->abort_flag;

  if (tid == 0) {
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(smem_u32(&hdr->full[s]), kProdWarps);
      mbar_init(smem_u32(&hdr->empty[s]), 1);
    }
    for (int b = 0; b < kAccs; ++b) {
      mbar_init(smem_u32(&hdr->acc_full[b]), 1);
      mbar_init(smem_u32(&hdr->acc_empty[b]), kEpiWarps);
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
    tmem_alloc(smem_u32(&hdr->tmem_base), tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = hdr->tmem_base;

  if (!p.after_own) pdl_wait();
  if (hdr->abort_flag != 0u) {
    pdl_wait();                                          // (and fall through to the common exit)
  } else if (warp < kProdWarps) {
    // =========================== producers ===========================
    if (LONG) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kLongProdRegs));
    const char* A = static_cast<const char*>(p.A);
    const char* Bs = static_cast<const char*>(p.Bsrc);
    const long long pitch_c = static_cast<long long>(p.C) * 4, pitch_n = static_cast<long long>(p.N) * 4;
    // Chunks of this thread, the same in every step: tid + 512 j of the A tile and of the B tile.  Tiles whose rows are M / N
    // indices (A of G and S, weights stored [n][contraction]) count eight chunks per row; tiles whose rows are 32 contraction
    // elements (weights [contraction][n], both tiles of D) count along rows of 32 or BN / 4 chunks.
    const bool b_rows_n = OP != kOpDweight && p.nc;
    const int cpr = p.BN / 4, b_chunks = p.BN * 8;
    const int cc = tid & 7, r0 = tid >> 3;             // chunk and row (+ 64 j) of the first kind
    const bool b_on[2] = {tid < b_chunks, tid + kProdThreads < b_chunks};
    int wr[2], wc[2];                                  // row and chunk of B, second kind
    uint32_t a_dst[2], b_dst[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      wr[j] = (tid + kProdThreads * j) / cpr;
      wc[j] = (tid + kProdThreads * j) - wr[j] * cpr;
      const int ar = OP == kOpDweight ? warp + kProdWarps * j : r0 + 64 * j;
      a_dst[j] = static_cast<uint32_t>(ar) * 128u +
                 (OP == kOpDweight ? static_cast<uint32_t>(lane >> 3) * (kStepElems * 128u) + swz32(lane, ar) : swz16(cc, ar));
      b_dst[j] = kATile + (b_rows_n ? static_cast<uint32_t>(r0 + 64 * j) * 128u + swz16(cc, r0)
                                    : static_cast<uint32_t>(wc[j] >> 3) * (kStepElems * 128u) + static_cast<uint32_t>(wr[j]) * 128u +
                                          swz32(wc[j], wr[j]));
    }

    // ---- load cursor: the unit and step the next issue belongs to ----
    int lu = blockIdx.x, lk = 0, lsteps = 0;
    Unit u{};
    const char* a_src[2];            // G, S: source of this thread's chunks in the step to issue, NULL = masked
    const char* b_src[2];
    // D: lane r of every warp keeps row r of the next step - its slot row (-1 beyond the range) and token id, loaded a step ahead
    // and looked at only when the step is issued; the other lanes get them by shuffles (one division and one load per lane)
    int row_slot = -1, row_b = 0;
    long long row_t = 0;
    auto look_up = [&](int k) {
      const int r = k * kStepElems + lane, m = u.split * p.rows_per_split + r;
      const bool on = r < p.rows_per_split && m < p.M;
      row_b = on ? m / p.K : 0;
      const int slot = (row_b * p.E + u.e) * p.K + (on ? m - row_b * p.K : 0);
      row_t = load_index(p.Ind, p.index_dtype, slot);
      row_slot = on ? slot : -1;
    };
    // G: token ids of the next unit's rows, loaded a unit ahead and looked at only when that unit begins
    long long ahead_t[2];
    auto fetch_ids = [&](int v) {
      const Unit w = unit_of<OP>(p, v);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int m = min(w.m0 + r0 + 64 * i, p.M - 1), b = m / p.K;
        ahead_t[i] = load_index(p.Ind, p.index_dtype, static_cast<long long>(b * p.E + w.e) * p.K + (m - b * p.K));
      }
    };
    auto begin_unit = [&]() {
      u = unit_of<OP>(p, lu);
      lsteps = unit_steps<OP>(p, u);
      lk = 0;
      if (OP == kOpDweight) {
        look_up(0);
        return;
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int m = u.m0 + r0 + 64 * i, b = m / p.K;
        int row = -1;
        if (OP == kOpScatter) row = m < p.M ? (b * p.E + u.e) * p.K + (m - b * p.K) : -1;
        else if (m < p.M && ahead_t[i] >= 0 && ahead_t[i] < p.T) row = b * p.T + static_cast<int>(ahead_t[i]);
        a_src[i] = row >= 0 ? A + static_cast<long long>(row) * pitch_c + cc * 16 : nullptr;
        b_src[i] = nullptr;
        if (b_rows_n) {
          if (u.n0 + r0 + 64 * i < p.N) b_src[i] = Bs + (static_cast<long long>(u.e) * p.N + u.n0 + r0 + 64 * i) * pitch_c + cc * 16;
        } else if (static_cast<long long>(u.n0) * 4 + wc[i] * 16 < pitch_n) {
          b_src[i] = Bs + (static_cast<long long>(u.e) * p.C + wr[i]) * pitch_n + static_cast<long long>(u.n0) * 4 + wc[i] * 16;
        }
      }
      if (OP == kOpGather && lu + static_cast<int>(gridDim.x) < p.units) fetch_ids(lu + gridDim.x);
    };
    const long long b_step = b_rows_n ? 128 : kStepElems * pitch_n;      // from one step to the next
    auto issue = [&](uint32_t base) {
      if (OP == kOpDweight) {
        const bool known = row_slot >= 0 && row_t >= 0 && row_t < p.T;
        if (row_slot >= 0 && !known && warp == 0 && u.m0 == 0 && u.n0 == 0) p.status.report(EGS_STATUS_INDEX_OUT_OF_RANGE);
        const int tok = known ? row_b * p.T + static_cast<int>(row_t) : -1;
        const bool a_col = static_cast<long long>(u.m0) * 4 + lane * 16 < pitch_c;
        const char* a_col_src = A + static_cast<long long>(u.m0) * 4 + lane * 16;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int tk = __shfl_sync(0xffffffffu, tok, warp + kProdWarps * i);
          const bool v = a_col && tk >= 0;
          cp_async16(base + a_dst[i], v ? a_col_src + tk * pitch_c : A, v ? 16u : 0u);
        }
        const char* b_col_src = Bs + static_cast<long long>(u.n0) * 4;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int slot = __shfl_sync(0xffffffffu, row_slot, wr[j] & 31);
          if (!b_on[j]) continue;
          const bool v = slot >= 0 && static_cast<long long>(u.n0) * 4 + wc[j] * 16 < pitch_n;
          cp_async16(base + b_dst[j], v ? b_col_src + slot * pitch_n + wc[j] * 16 : Bs, v ? 16u : 0u);
        }
        if (lk + 1 < lsteps) look_up(lk + 1);
        return;
      }
      const int k0 = lk * kStepElems;
      const bool kvalid = k0 + cc * 4 < p.C;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const bool v = kvalid && a_src[i];
        cp_async16(base + a_dst[i], v ? a_src[i] : A, v ? 16u : 0u);
        if (a_src[i]) a_src[i] += 128;
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (!b_on[j]) continue;
        const bool v = b_src[j] && (b_rows_n ? kvalid : k0 + wr[j] < p.C);
        cp_async16(base + b_dst[j], v ? b_src[j] : Bs, v ? 16u : 0u);
        if (b_src[j]) b_src[j] += b_step;
      }
    };
    auto issue_next = [&](int slot) {          // the next step of this CTA's sequence, if there is one
      if (lu < p.units) {
        issue(raw0 + static_cast<uint32_t>(slot) * stage_bytes);
        if (++lk == lsteps) {
          lu += gridDim.x;
          if (lu < p.units) begin_unit();
        }
      }
      cp_async_commit();
    };

    int total = 0;                             // steps of this CTA
    for (int v = blockIdx.x; v < p.units; v += gridDim.x) total += unit_steps<OP>(p, unit_of<OP>(p, v));
    const int dist = raw - kLoStages;
    if (lu < p.units) {
      if (OP == kOpGather) fetch_ids(lu);
      begin_unit();
    }
    for (int g = 0; g < dist; ++g) issue_next(g);
    bool alive = true;
    int slot = 0, ahead = dist;                // raw slot of step g, and of step g + dist
    int eslot = 0, eround = 0;                 // barrier slot and round of step g - kLoStages
    for (int g = 0; g < total && alive; ++g) {
      cp_async_wait_pending(dist - 1);
      if (g >= kLoStages) {
        alive = mbar_wait_all(smem_u32(&hdr->empty[eslot]), eround & 1, abort_flag, p.status.word);
        if (!alive) break;
        if (++eslot == raw) { eslot = 0; ++eround; }
      }
      const uint32_t src = raw0 + static_cast<uint32_t>(slot) * stage_bytes;
      const uint32_t dst = lo0 + static_cast<uint32_t>(g & (kLoStages - 1)) * stage_bytes;
      uint4 xa[2], xb[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) xa[i] = load_chunk(src + a_dst[i]);
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (b_on[j]) xb[j] = load_chunk(src + b_dst[j]);
#pragma unroll
      for (int i = 0; i < 2; ++i) store_lo(dst + a_dst[i], xa[i]);
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (b_on[j]) store_lo(dst + b_dst[j], xb[j]);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&hdr->full[slot]));
      if (++slot == raw) slot = 0;
      issue_next(ahead);                       // its slot is the one step g - kLoStages has left
      if (++ahead == raw) ahead = 0;
    }
    cp_async_wait_all();
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
    for (int un = blockIdx.x; un < p.units && alive; un += gridDim.x) {
      const Unit u = unit_of<OP>(p, un);
      const int steps = unit_steps<OP>(p, u);
      int my_ro = -1;                                    // G, S: destination row of tile row lg * 32 + lane
      if (OP != kOpDweight) {
        const int m = u.m0 + lg * 32 + lane;
        if (m < p.M) {
          const int b = m / p.K, k = m - b * p.K;
          const int slot = (b * p.E + u.e) * p.K + k;
          const long long tk = load_index(p.Ind, p.index_dtype, slot);
          const bool ok = tk >= 0 && tk < p.T;
          if (!ok && u.n0 == 0) p.status.report(EGS_STATUS_INDEX_OUT_OF_RANGE);
          my_ro = OP == kOpGather ? slot : (ok ? b * p.T + static_cast<int>(tk) : -1);
        }
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
        uint32_t v[kBlocks][32];                         // the sums of this thread's row
        for (int ch = 0; ch < steps; ++ch) {
          const uint32_t acc = wait_full();
          if (!alive) break;
#pragma unroll
          for (int c = 0; c < kBlocks; ++c) {
            if (c * kShares + share < nblk) {
              uint32_t x[32];
              tmem_ld32(acc + static_cast<uint32_t>((c * kShares + share) * 32), x);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; i += 2) {
                if (ch == 0) {
                  v[c][i] = x[i];
                  v[c][i + 1] = x[i + 1];
                } else {
                  add2(v[c][i], v[c][i + 1], x[i], x[i + 1]);
                }
              }
            }
          }
          release();
        }
        if (!alive) break;
#pragma unroll
        for (int c = 0; c < kBlocks; ++c) {
          if (c * kShares + share < nblk) {
            again_if_nan(c * kShares + share, v[c]);
            emit(c * kShares + share, v[c]);
          }
        }
      } else {
        const uint32_t acc = wait_full();
        if (!alive) break;
        for (int c = 0; c < nblk; ++c) {
          uint32_t v[32];
          tmem_ld32(acc + static_cast<uint32_t>(c * 32), v);
          tmem_ld_wait();
          emit(c, v);
        }
        release();
      }
    }
  } else {
    // =========================== MMA issuer ===========================
    if (LONG) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kLongMmaRegs));
    // (the warp runs converged and an elected lane issues, see mbar_wait_all: twelve MMAs from a lane on its own took 1000 clocks)
    // A: K-major rows (G, S) or rows = contraction (D); B: rows = n (weights [n][contraction]) or rows = contraction
    const bool a_mn = OP == kOpDweight, b_mn = OP == kOpDweight || !p.nc;
    const uint32_t a_lbo = a_mn ? kStepElems * 128u : 16u, a_sbo = a_mn ? 512u : 1024u, a_lay = a_mn ? kSwizzle128Base32 : kSwizzle128;
    const uint32_t b_lbo = b_mn ? kStepElems * 128u : 16u, b_sbo = b_mn ? 512u : 1024u, b_lay = b_mn ? kSwizzle128Base32 : kSwizzle128;
    const uint32_t a_adv = (a_mn ? 8u * 128u : 32u) >> 4, b_adv = (b_mn ? 8u * 128u : 32u) >> 4;
    const uint64_t a_desc = make_smem_desc(0u, a_lbo, a_sbo, a_lay), b_desc = make_smem_desc(0u, b_lbo, b_sbo, b_lay) + (kATile >> 4);
    bool ok = true;
    int buf = 0, around = 0, slot = 0, round = 0, lo = 0;
    for (int un = blockIdx.x; un < p.units && ok && warp == kMmaWarp; un += gridDim.x) {
      const Unit u = unit_of<OP>(p, un);
      const int steps = unit_steps<OP>(p, u);
      const int bn = min(p.BN, ((p.N - u.n0) + 15) & ~15);
      const uint32_t idesc = make_idesc(2u, a_mn ? 1u : 0u, b_mn ? 1u : 0u, kTileM, static_cast<uint32_t>(bn));
      // contraction elements of the unit (rows for D)
      const int len = OP == kOpDweight ? min(p.rows_per_split, p.M - u.split * p.rows_per_split) : p.C;
      for (int ks = 0; ks < steps && ok; ++ks) {
        const bool first = LONG || ks == 0, last = LONG || ks == steps - 1;
        if (first && around > 0) {
          ok = mbar_wait_all(smem_u32(&hdr->acc_empty[buf]), (around - 1) & 1, abort_flag, p.status.word);
          if (!ok) break;
        }
        ok = mbar_wait_all(smem_u32(&hdr->full[slot]), round & 1, abort_flag, p.status.word);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d = tmem_base + static_cast<uint32_t>(buf) * acc_cols;
        // (descriptors: 14 address bits in 16-byte units; shared memory is smaller)
        const uint32_t hi16 = (raw0 + static_cast<uint32_t>(slot) * stage_bytes) >> 4, lo16 = (lo0 + static_cast<uint32_t>(lo) * stage_bytes) >> 4;
        const int nkq = min(4, (len - ks * kStepElems + 7) / 8);
        if (elect_one()) {
          auto hi_hi = [&](int kq) { umma<true>(d, a_desc + (hi16 + kq * a_adv), b_desc + (hi16 + kq * b_adv), idesc, 1u); };
#pragma unroll
          for (int kq = 0; kq < 4; ++kq) {
            if (kq < nkq) {
              umma<true>(d, a_desc + (lo16 + kq * a_adv), b_desc + (hi16 + kq * b_adv), idesc, (first && kq == 0) ? 0u : 1u);
              umma<true>(d, a_desc + (hi16 + kq * a_adv), b_desc + (lo16 + kq * b_adv), idesc, 1u);
              if (!LONG) hi_hi(kq);
            }
          }
          if (LONG) {                                    // the small products first: additions truncate, and to a small sum that is little
#pragma unroll
            for (int kq = 0; kq < 4; ++kq)
              if (kq < nkq) hi_hi(kq);
          }
          umma_commit(smem_u32(&hdr->empty[slot]));
          if (last) umma_commit(smem_u32(&hdr->acc_full[buf]));
        }
        if (last && ++buf == kAccs) { buf = 0; ++around; }
        lo ^= 1;
        if (++slot == raw) { slot = 0; ++round; }
      }
    }
    pdl_trigger();                                       // (not before: a dependent's waiting CTAs would keep a kernel of another stream off this SM)
    __syncwarp();
  }

  // ---- common exit ----
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) tmem_release(tmem_base, tmem_cols, smem_u32(&hdr->drain), abort_flag, p.status, lane);
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
int strict_raw_stages(int bn, bool long_c) {
  const size_t stage = kATile + static_cast<size_t>(bn) * 128;
  size_t raw = (kSmemMax - kStrictHeader - xpose_bytes(long_c)) / stage - kLoStages;
  return static_cast<int>(raw > kMaxStages ? kMaxStages : raw);
}

template <int OP, bool LONG = false>
cudaError_t launch(const StrictParams& p, cudaStream_t st) {
  const size_t stage = kATile + static_cast<size_t>(p.BN) * 128;
  const size_t smem = kStrictHeader + xpose_bytes(LONG) + (p.raw + kLoStages) * stage;
  cudaError_t err = ensure_smem_optin<strict_kernel<OP, LONG>>(static_cast<int>(kSmemMax));
  if (err != cudaSuccess) return err;
  if (LONG) {                                            // setmaxnreg can only share out what the block is launched with
    static const int regs = [] {
      cudaFuncAttributes a{};
      return cudaFuncGetAttributes(&a, strict_kernel<OP, LONG>) == cudaSuccess ? a.numRegs : 0;
    }();
    if (regs * strict_threads(true) < (kProdWarps * kLongProdRegs + epi_warps(true) * kLongEpiRegs + 4 * kLongMmaRegs) * 32) return cudaErrorInvalidConfiguration;
  }
  err = launch_kernel(strict_kernel<OP, LONG>, p.units < kSms ? p.units : kSms, strict_threads(LONG), smem, st, true, p);
  count_launch();
  return err;
}

}  // namespace

void configure_strict_rowgemm(RowGemmParams& p) {
  p.BN = strict_bn(p.N);
  p.stages = strict_raw_stages(p.BN, long_contraction(p.C));
  p.row_tiles = 1;
  p.persistent = 1;
}

cudaError_t launch_strict_rowgemm(const RowGemmParams& r, bool scatter, cudaStream_t st) {
  StrictParams p{};
  p.A = r.A; p.Bsrc = r.W; p.bias = r.bias; p.Ind = r.Ind; p.Out = static_cast<float*>(r.Out); p.status = r.status;
  p.B = r.B; p.T = r.T; p.E = r.E; p.K = r.K; p.M = r.M; p.C = r.C; p.N = r.N;
  p.nc = r.w_layout == EGS_W_NC;
  p.index_dtype = r.index_dtype;
  p.BN = r.BN; p.raw = r.stages;
  p.after_own = r.after_own;
  p.tiles_m = (r.M + kTileM - 1) / kTileM;
  p.tiles_n = (r.N + r.BN - 1) / r.BN;
  const long long units = static_cast<long long>(p.tiles_m) * p.tiles_n * p.E;
  if (units > 2147483647ll) return cudaErrorInvalidValue;
  p.units = static_cast<int>(units);
  if (long_contraction(r.C))
    return scatter ? launch<kOpScatter, true>(p, st) : launch<kOpGather, true>(p, st);
  return scatter ? launch<kOpScatter>(p, st) : launch<kOpGather>(p, st);
}

void configure_strict_dweight(DWeightParams& p) {
  p.BN = strict_bn(p.FD);
  p.stages = strict_raw_stages(p.BN, false);
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
  p.BN = r.BN; p.raw = r.stages;
  p.after_own = r.after_own;
  p.splits = r.splits; p.rows_per_split = r.rows_per_split;
  p.tiles_m = (r.FG + kTileM - 1) / kTileM;
  p.tiles_n = (r.FD + r.BN - 1) / r.BN;
  const long long units = static_cast<long long>(p.tiles_m) * p.tiles_n * p.E * p.splits;
  if (units > 2147483647ll) return cudaErrorInvalidValue;
  p.units = static_cast<int>(units);
  return launch<kOpDweight>(p, st);
}

}  // namespace egs

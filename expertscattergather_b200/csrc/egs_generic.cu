// Generic CUDA-core kernels for the three operators: any sizes, any alignment, fp32 accumulation.
// They serve shapes the tensor-core kernels do not take (row pitches that are not multiples of
// 16 bytes, e.g. the odd dimensions the reference's tests draw, test_all.py:98) and are the
// on-device cross-check for the tensor-core family.  Also here: the zero-fill and fp32->dtype
// conversion kernels.
#include "egs_internal.cuh"

namespace egs {

namespace {

// The row kernel and the first weight-gradient kernel: 128 threads as 16 (ty) x 8 (tx), operands converted to float32 in shared memory, contraction steps of 32.
// What bounds them is the chain of a step - load, barrier, multiply - so the next step's elements are fetched into registers
// while the current one is multiplied, lanes run along the contiguous direction of every row (whole 128-byte segments), and
// several CTAs share an SM.  Results leave through shared memory for the same reason: rows are written (or added to) 32
// consecutive elements per instruction.  Tile widths are multiples of 32 chosen on the host so that little of a tile is
// padding: the widths that come here are mostly odd and below 128.
// Products go two at a time (fma.rn.f32x2, each rounded like fmaf: the same bits): 77880 rows 101 -> 101 82 -> 74 us, 100000 rows 127 -> 63
// 49 -> 41 us.  (Eight rows a thread, 64 threads a CTA and a ring of three cp.async stages read shared memory less and took 84 and 49:
// there is more to gain from CTAs in flight, whose chain is id, row, product, store.)
// These kernels, the fills before them and the conversions after them do not trigger their dependents: those start when they have left.
// CTAs of which an SM holds several settle on the SMs that the kernel before them leaves first, and stay there: a scatter of 48 CTAs
// behind its fill (float32, 200 rows of 333 to 701 features for each of 2 experts) took 34 us with triggers at the start, 27
// without dependent launches, 23 so; the operators of a training pass at 46 rows, 1025 and 305 features, 10 experts 233, 245 and 217 (265 with
// triggers where the results are written), at 595 rows, 139 and 187, 11 experts 154, 155 and 127.
// 54855 routed rows, 83 -> 29 features, float32 (gather): 13 us; 45 us with fixed 64x64x16 tiles and no prefetch.
constexpr int NTHREADS = 128;
constexpr int TM = 64;          // rows per CTA of the row kernel
constexpr int TK = 32;          // contraction step
constexpr int APITCH = TK + 4;  // floats; rows 16-byte aligned, consecutive rows 4 banks apart

// two products at a time
__device__ __forceinline__ unsigned long long pair_of(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ float4 float4_of(unsigned long long a, unsigned long long b) {
  float4 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.z), "=f"(r.w) : "l"(b));
  return r;
}

// ------------------------------------------------------------------------------------------------
// G and S:  tile[m, n] = sum_c A[row_a(m), c] * W(e, c, n);   G stores it, S adds it atomically
// (operator G: egs/triton_kernels.py:48-143, operator S: :156-247 in the reference)
// NJ: tile width in units of 32 columns.  Thread (ty, tx) owns rows ty + 16 i and columns 32 j + 4 tx .. + 3.
// ------------------------------------------------------------------------------------------------
// CTAS: CTAs that share an SM.  96 columns spill at four (float32), and a contraction of several steps pays for that: 32768 rows 1001 -> 257 of 16 experts
// 549 us with four, 546 before products went in pairs, 483 with three; 960 rows 655 -> 67 70, 59 and 51.  A single step is over too soon: 60680 rows
// 5 -> 177 24 us with four, 26 with three.
template <typename T, bool SCATTER, int NJ, int CTAS>
__global__ void __launch_bounds__(NTHREADS, CTAS) generic_rowgemm_kernel(RowGemmParams p) {
  constexpr int BN = 32 * NJ, BPITCH = BN + 4;
  __shared__ __align__(16) float As[TM * APITCH];
  __shared__ __align__(16) float Bs[TK * BPITCH];
  __shared__ long long row_a[TM];   // element offset of the A row, -1 when masked
  __shared__ long long row_o[TM];   // element offset of the output row, -1 when masked

  const int e = blockIdx.z;
  const int m0 = blockIdx.x * TM;
  const int n0 = blockIdx.y * BN;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tx = tid & 7, ty = tid >> 3;
  pdl_wait();
  const T* A = static_cast<const T*>(p.A);
  const T* W = static_cast<const T*>(p.W) + static_cast<long long>(e) * p.C * p.N;
  T* Out = static_cast<T*>(p.Out);

  if (tid < TM) {
    const int m = m0 + tid;
    long long ra = -1, ro = -1;
    if (m < p.M) {
      const int b = m / p.K, k = m - b * p.K;
      const long long slot = (static_cast<long long>(b) * p.E + e) * p.K + k;
      const long long t = load_index(p.Ind, p.index_dtype, slot);
      if (t >= 0 && t < p.T) {
        const long long tok = static_cast<long long>(b) * p.T + t;
        ra = (SCATTER ? slot : tok) * p.C;
        ro = (SCATTER ? tok : slot) * p.N;
      } else {
        p.status.report(EGS_STATUS_INDEX_OUT_OF_RANGE);
        if (!SCATTER) ro = slot * p.N;   // gather: the row is still written (zeros)
      }
    }
    row_a[tid] = ra;
    row_o[tid] = ro;
  }
  __syncthreads();

  float ra[TM / 4], rb[8 * NJ];
  auto fetch = [&](int c0) {
    const int c = c0 + lane;
#pragma unroll
    for (int i = 0; i < TM / 4; ++i) {
      const long long off = row_a[warp + 4 * i];
      ra[i] = (off >= 0 && c < p.C) ? to_f32<T>(A[off + c]) : 0.f;
    }
    if (p.w_layout == EGS_W_CN) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int cc = c0 + warp + 4 * i;
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const int n = n0 + 32 * j + lane;
          rb[i * NJ + j] = (cc < p.C && n < p.N) ? to_f32<T>(W[static_cast<long long>(cc) * p.N + n]) : 0.f;
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8 * NJ; ++i) {
        const int n = n0 + warp + 4 * i;
        rb[i] = (c < p.C && n < p.N) ? to_f32<T>(W[static_cast<long long>(n) * p.C + c]) : 0.f;
      }
    }
  };
  auto stage = [&]() {
#pragma unroll
    for (int i = 0; i < TM / 4; ++i) As[(warp + 4 * i) * APITCH + lane] = ra[i];
    if (p.w_layout == EGS_W_CN) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) Bs[(warp + 4 * i) * BPITCH + 32 * j + lane] = rb[i * NJ + j];
    } else {
#pragma unroll
      for (int i = 0; i < 8 * NJ; ++i) Bs[lane * BPITCH + warp + 4 * i] = rb[i];
    }
  };

  unsigned long long acc[4][2 * NJ] = {};
  fetch(0);
  for (int c0 = 0; c0 < p.C; c0 += TK) {
    stage();
    __syncthreads();
    if (c0 + TK < p.C) fetch(c0 + TK);
#pragma unroll 1
    for (int kk = 0; kk < TK; kk += 4) {
      if (c0 + kk >= p.C) break;
      float4 a[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(&As[(ty + 16 * i) * APITCH + kk]);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(&Bs[(kk + q) * BPITCH + 32 * j + 4 * tx]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float av = q == 0 ? a[i].x : q == 1 ? a[i].y : q == 2 ? a[i].z : a[i].w;
            const unsigned long long aa = pair_of(av, av);
            fma2(acc[i][2 * j], aa, b.x);
            fma2(acc[i][2 * j + 1], aa, b.y);
          }
        }
      }
    }
    __syncthreads();
  }

  // 32 columns at a time through As: lanes then cover 32 consecutive elements of one row
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    if (n0 + 32 * j >= p.N) break;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<float4*>(&As[(ty + 16 * i) * APITCH + 4 * tx]) =
          float4_of(acc[i][2 * j], acc[i][2 * j + 1]);
    __syncthreads();
    const int n = n0 + 32 * j + lane;
    if (n < p.N) {
      const float bias = p.bias ? to_f32<T>(static_cast<const T*>(p.bias)[static_cast<long long>(e) * p.N + n]) : 0.f;
#pragma unroll 4
      for (int r = warp; r < TM; r += 4) {
        const long long ro = row_o[r];
        if (ro < 0) continue;
        const float v = As[r * APITCH + lane] + bias;
        if (SCATTER) {
          if (sizeof(T) == 2) atomicAdd(p.acc + ro + n, v);   // 16-bit: float32 accumulation rows
          else atomicAdd(reinterpret_cast<float*>(Out) + ro + n, v);
        } else {
          Out[ro + n] = from_f32<T>(v);
        }
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------------------
// D:  P[e, f, g] = sum_m Xsrc[token row(m), f] * Ysrc[slot row(m), g]
// (operator D: egs/triton_kernels.py:261-356 in the reference)
// FI, GJ: tile size in units of 32 gathered / direct features.  Thread (ty, tx) owns features f = 32 i + 2 ty + {0, 1} and
// g = 32 j + 4 tx .. + 3.  A tile is summed over `rows_per_split` rows and added to the float32 result where there are several.
// For up to 32 direct features, and for wider ones of float32 where there are few CTAs; else the kernel after this.
// ------------------------------------------------------------------------------------------------
constexpr int kRowTable = 256;   // rows whose offsets are looked up at a time
template <typename T, int FI, int GJ>
__global__ void __launch_bounds__(NTHREADS, FI * GJ > 4 ? 3 : 4) generic_dweight_kernel(DWeightParams p) {
  constexpr int FP = 32 * FI + 4, GP = 32 * GJ + 4, XP = 33;
  constexpr int kTile = TK * (FP + GP) > 32 * XP ? TK * (FP + GP) : 32 * XP;
  __shared__ __align__(16) float tile[kTile];
  __shared__ long long row_g[kRowTable];
  __shared__ long long row_d[kRowTable];
  float* Fs = tile;
  float* Gs = tile + TK * FP;

  const int e = blockIdx.z / p.splits;
  const int split = blockIdx.z - e * p.splits;
  const int f0 = blockIdx.x * 32 * FI;
  const int g0 = blockIdx.y * 32 * GJ;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tx = tid & 7, ty = tid >> 3;
  pdl_wait();
  const T* Xs = static_cast<const T*>(p.Xsrc);
  const T* Ys = static_cast<const T*>(p.Ysrc);

  const int m_begin = split * p.rows_per_split;
  const int m_end = min(p.M, m_begin + p.rows_per_split);
  float acc[2 * FI][4 * GJ] = {};
  float rf[8 * FI], rg[8 * GJ];
  auto fetch = [&](int r0) {       // r0: first row of the step within the table
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const long long og = row_g[r0 + warp + 4 * k], od = row_d[r0 + warp + 4 * k];
#pragma unroll
      for (int i = 0; i < FI; ++i) {
        const int f = f0 + 32 * i + lane;
        rf[k * FI + i] = (og >= 0 && f < p.FG) ? to_f32<T>(Xs[og + f]) : 0.f;
      }
#pragma unroll
      for (int j = 0; j < GJ; ++j) {
        const int g = g0 + 32 * j + lane;
        rg[k * GJ + j] = (od >= 0 && g < p.FD) ? to_f32<T>(Ys[od + g]) : 0.f;
      }
    }
  };

  for (int mt = m_begin; mt < m_end; mt += kRowTable) {
    __syncthreads();
    for (int i = tid; i < kRowTable; i += NTHREADS) {
      const int m = mt + i;
      long long og = -1, od = -1;
      if (m < m_end) {
        const int b = m / p.K, k = m - b * p.K;
        const long long slot = (static_cast<long long>(b) * p.E + e) * p.K + k;
        const long long t = load_index(p.Ind, p.index_dtype, slot);
        if (t >= 0 && t < p.T) {
          og = (static_cast<long long>(b) * p.T + t) * p.FG;
          od = slot * p.FD;
        } else {
          p.status.report(EGS_STATUS_INDEX_OUT_OF_RANGE);
        }
      }
      row_g[i] = og;
      row_d[i] = od;
    }
    __syncthreads();
    const int nrows = min(kRowTable, m_end - mt);
    fetch(0);
    for (int r0 = 0; r0 < nrows; r0 += TK) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
#pragma unroll
        for (int i = 0; i < FI; ++i) Fs[(warp + 4 * k) * FP + 32 * i + lane] = rf[k * FI + i];
#pragma unroll
        for (int j = 0; j < GJ; ++j) Gs[(warp + 4 * k) * GP + 32 * j + lane] = rg[k * GJ + j];
      }
      __syncthreads();
      if (r0 + TK < nrows) fetch(r0 + TK);
#pragma unroll 4
      for (int kk = 0; kk < TK; ++kk) {
        float2 a[FI];
        float4 b[GJ];
#pragma unroll
        for (int i = 0; i < FI; ++i) a[i] = *reinterpret_cast<const float2*>(&Fs[kk * FP + 32 * i + 2 * ty]);
#pragma unroll
        for (int j = 0; j < GJ; ++j) b[j] = *reinterpret_cast<const float4*>(&Gs[kk * GP + 32 * j + 4 * tx]);
#pragma unroll
        for (int i = 0; i < FI; ++i)
#pragma unroll
          for (int j = 0; j < GJ; ++j) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const float av = u ? a[i].y : a[i].x;
              acc[2 * i + u][4 * j] = fmaf(av, b[j].x, acc[2 * i + u][4 * j]);
              acc[2 * i + u][4 * j + 1] = fmaf(av, b[j].y, acc[2 * i + u][4 * j + 1]);
              acc[2 * i + u][4 * j + 2] = fmaf(av, b[j].z, acc[2 * i + u][4 * j + 2]);
              acc[2 * i + u][4 * j + 3] = fmaf(av, b[j].w, acc[2 * i + u][4 * j + 3]);
            }
          }
      }
      __syncthreads();
    }
  }

  // 32 x 32 blocks through shared memory, lanes along the contiguous direction of the output
  T* out = static_cast<T*>(p.out);
  const bool fg = p.out_layout == EGS_DW_GATHERED_ROWS;
#pragma unroll
  for (int i = 0; i < FI; ++i)
#pragma unroll
    for (int j = 0; j < GJ; ++j) {
      if (f0 + 32 * i >= p.FG || g0 + 32 * j >= p.FD) continue;
      __syncthreads();
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) tile[(2 * ty + u) * XP + 4 * tx + v] = acc[2 * i + u][4 * j + v];
      __syncthreads();
#pragma unroll
      for (int r = warp; r < 32; r += 4) {
        const int f = f0 + 32 * i + (fg ? r : lane), g = g0 + 32 * j + (fg ? lane : r);
        if (f < p.FG && g < p.FD) {
          const float v = fg ? tile[r * XP + lane] : tile[lane * XP + r];
          const long long off = fg ? (static_cast<long long>(e) * p.FG + f) * p.FD + g : (static_cast<long long>(e) * p.FD + g) * p.FG + f;
          if (p.splits > 1) atomicAdd(p.acc + off, v);
          else out[off] = from_f32<T>(v);
        }
      }
    }
}

// ------------------------------------------------------------------------------------------------
// D for more than 32 direct features: 64 threads as 8 (ty) x 8 (tx), each with features f = 32 i + 4 ty .. + 3 and g = 32 j + 4 tx .. + 3.
// Twice the products of a thread of the kernel above for half as many more loads from shared memory.  Shared memory is a ring of three
// stages of 16 rows (two: 3 % slower); the rows two steps ahead are loaded into registers before the products of a step and stored
// behind them.  Loaded, converted and stored at once, 16-bit types waited for memory in every step: 271 us for 79200 rows 101 x 101 in bf16, where
// the kernel above takes 185 and this one 99.  4-byte cp.async, for float32 only, took 58 us at 100000 rows 127 x 63 and 95 at 196416
// rows 111 x 33, this one 54 and 87, the kernel above 74 and 126.
// Two warps keep two of an SM's four schedulers busy, so a float32 grid of less than two CTAs an SM takes the kernel above: 1416 rows
// 107 x 119 12.6 us there and 17.7 here, 3212 of 1 x 63 6.8 and 8.8; from there on this one is the faster (15048 rows 25 x 557: 38 and 26), and for
// 16-bit types always (1584 rows 95 x 445: 21.8 and 19.4, 3807 of 39 x 55 15.4 and 13.3).
// ------------------------------------------------------------------------------------------------
constexpr int kWideThreads = 64, kWideStep = 16, kWideStages = 3;

template <typename T, int FI, int GJ>
__global__ void __launch_bounds__(kWideThreads, FI > 2 ? 4 : FI > 1 ? 5 : 8) generic_dweight_wide_kernel(DWeightParams p) {
  constexpr int FP = 32 * FI + 4, GP = 32 * GJ + 4, XP = 33;
  __shared__ __align__(16) float tile[kWideStages * kWideStep * (FP + GP)];
  __shared__ long long row_g[kRowTable];
  __shared__ long long row_d[kRowTable];
  static_assert(32 * XP <= kWideStages * kWideStep * (FP + GP), "the read-out goes through the ring");

  const int e = blockIdx.z / p.splits;
  const int split = blockIdx.z - e * p.splits;
  const int f0 = blockIdx.x * 32 * FI;
  const int g0 = blockIdx.y * 32 * GJ;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tx = tid & 7, ty = tid >> 3;
  pdl_wait();
  const T* Xs = static_cast<const T*>(p.Xsrc);
  const T* Ys = static_cast<const T*>(p.Ysrc);

  const int m_begin = split * p.rows_per_split;
  const int m_end = min(p.M, m_begin + p.rows_per_split);
  unsigned long long acc[4 * FI][2 * GJ] = {};
  constexpr int kRows = kWideStep / 2;
  T held[kRows][FI + GJ];
  auto load = [&](int step) {      // this thread's elements of a step of the rows in the table, zero where they are masked
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      const int r = step * kWideStep + warp + 2 * k;
      const long long og = row_g[r], od = row_d[r];
#pragma unroll
      for (int i = 0; i < FI; ++i) {
        const int f = f0 + 32 * i + lane;
        held[k][i] = og >= 0 && f < p.FG ? Xs[og + f] : from_f32<T>(0.f);
      }
#pragma unroll
      for (int j = 0; j < GJ; ++j) {
        const int g = g0 + 32 * j + lane;
        held[k][FI + j] = od >= 0 && g < p.FD ? Ys[od + g] : from_f32<T>(0.f);
      }
    }
  };
  auto store = [&](int step) {
    float* F = tile + step % kWideStages * (kWideStep * (FP + GP));
    float* G = F + kWideStep * FP;
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      const int r = warp + 2 * k;
#pragma unroll
      for (int i = 0; i < FI; ++i) F[r * FP + 32 * i + lane] = to_f32<T>(held[k][i]);
#pragma unroll
      for (int j = 0; j < GJ; ++j) G[r * GP + 32 * j + lane] = to_f32<T>(held[k][FI + j]);
    }
  };

  for (int mt = m_begin; mt < m_end; mt += kRowTable) {
    __syncthreads();
#pragma unroll
    for (int i = tid; i < kRowTable; i += kWideThreads) {
      const int m = mt + i;
      long long og = -1, od = -1;
      if (m < m_end) {
        const int b = m / p.K, k = m - b * p.K;
        const long long slot = (static_cast<long long>(b) * p.E + e) * p.K + k;
        const long long t = load_index(p.Ind, p.index_dtype, slot);
        if (t >= 0 && t < p.T) {
          og = (static_cast<long long>(b) * p.T + t) * p.FG;
          od = slot * p.FD;
        } else {
          p.status.report(EGS_STATUS_INDEX_OUT_OF_RANGE);
        }
      }
      row_g[i] = og;
      row_d[i] = od;
    }
    __syncthreads();
    const int steps = (min(kRowTable, m_end - mt) + kWideStep - 1) / kWideStep;
#pragma unroll
    for (int s = 0; s < kWideStages - 1; ++s) {
      if (s < steps) {
        load(s);
        store(s);
      }
    }
    for (int s = 0; s < steps; ++s) {
      const int ahead = s + kWideStages - 1;             // (its stage was read in the step before this one)
      __syncthreads();
      if (ahead < steps) load(ahead);
      const float* F = tile + s % kWideStages * (kWideStep * (FP + GP)) + 4 * ty;
      const float* G = tile + s % kWideStages * (kWideStep * (FP + GP)) + kWideStep * FP + 4 * tx;
#pragma unroll 4
      for (int kk = 0; kk < kWideStep; ++kk) {
        float4 a[FI];
        ulonglong2 b[GJ];
#pragma unroll
        for (int i = 0; i < FI; ++i) a[i] = *reinterpret_cast<const float4*>(F + kk * FP + 32 * i);
#pragma unroll
        for (int j = 0; j < GJ; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(G + kk * GP + 32 * j);
#pragma unroll
        for (int i = 0; i < FI; ++i)
#pragma unroll
          for (int j = 0; j < GJ; ++j) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const float av = u == 0 ? a[i].x : u == 1 ? a[i].y : u == 2 ? a[i].z : a[i].w;
              const unsigned long long aa = pair_of(av, av);
              fma2(acc[4 * i + u][2 * j], aa, b[j].x);
              fma2(acc[4 * i + u][2 * j + 1], aa, b[j].y);
            }
          }
      }
      if (ahead < steps) store(ahead);
    }
  }

  // 32 x 32 blocks through shared memory, lanes along the contiguous direction of the output
  T* out = static_cast<T*>(p.out);
  const bool fg = p.out_layout == EGS_DW_GATHERED_ROWS;
#pragma unroll
  for (int i = 0; i < FI; ++i)
#pragma unroll
    for (int j = 0; j < GJ; ++j) {
      if (f0 + 32 * i >= p.FG || g0 + 32 * j >= p.FD) continue;
      __syncthreads();
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 x = float4_of(acc[4 * i + u][2 * j], acc[4 * i + u][2 * j + 1]);
        float* to = tile + (4 * ty + u) * XP + 4 * tx;
        to[0] = x.x;
        to[1] = x.y;
        to[2] = x.z;
        to[3] = x.w;
      }
      __syncthreads();
#pragma unroll 8
      for (int r = warp; r < 32; r += 2) {
        const int f = f0 + 32 * i + (fg ? r : lane), g = g0 + 32 * j + (fg ? lane : r);
        if (f < p.FG && g < p.FD) {
          const float v = fg ? tile[r * XP + lane] : tile[lane * XP + r];
          const long long off = fg ? (static_cast<long long>(e) * p.FG + f) * p.FD + g : (static_cast<long long>(e) * p.FD + g) * p.FG + f;
          if (p.splits > 1) atomicAdd(p.acc + off, v);
          else out[off] = from_f32<T>(v);
        }
      }
    }
}

// ------------------------------------------------------------------------------------------------
// Row sums per expert (the bias gradients):  out[e, n] = sum over the slots of expert e of row[n] of a token row (through Ind)
// or of the slot row itself (Ind == NULL).  Eight lanes cover 128 bytes of a row; a cluster of CTAs shares the rows of one
// (expert, 128-byte column block) and adds its partial sums through distributed shared memory, so that there is neither a
// scratch buffer nor a second pass and the order of the additions is fixed.  A thread adds eight rows as a tree and the trees with
// the rounding errors of their additions carried along (Knuth's TwoSum), and the threads' sums are added in 64 bits, so that long
// sums stay as good as short ones: 2^21 float32 rows of normal values to 1e-7, 2.4e-6 as one running sum.
// What bounds it are the loads: 65536 routed rows of 768 bf16 features in 16 us = 6.3 TB/s from L2 and HBM (40 us as the
// weight-gradient contraction against ones).
// ------------------------------------------------------------------------------------------------
constexpr int kSumThreads = 256;
template <typename T, bool VEC>
__global__ void __launch_bounds__(kSumThreads) expert_row_sum_kernel(const T* __restrict__ Src, const void* __restrict__ Ind,
                                                                     int index_dtype, T* __restrict__ out, int T_, int E, int K, int N,
                                                                     int M, int nranks, StatusRef status) {
  constexpr int PER = VEC ? 16 / static_cast<int>(sizeof(T)) : 1;   // columns per lane
  constexpr int COLS = 8 * PER;                                     // columns per CTA
  constexpr int ROWS = kSumThreads / 8;                             // rows a CTA reads at a time
  __shared__ float part[ROWS][COLS + 1];
  __shared__ double total[COLS];
  const int rank = blockIdx.x % nranks;                             // a cluster is `nranks` CTAs along x
  const int e = blockIdx.y, c0 = blockIdx.x / nranks * COLS;
  const int tid = threadIdx.x, cl = tid & 7, rl = tid >> 3;
  const int col = c0 + cl * PER;
  const int per = (M + nranks - 1) / nranks, m_end = min(M, (rank + 1) * per);
  float acc[PER], low[PER];                                         // running sums, and what rounding took from them
#pragma unroll
  for (int i = 0; i < PER; ++i) acc[i] = low[i] = 0.f;
  pdl_trigger();
  auto add = [&](int i, float t) {
    const float s = acc[i] + t, b = s - acc[i];
    low[i] += (acc[i] - (s - b)) + (t - b);
    acc[i] = s;
  };
  // eight rows in flight; each of a row's eight lanes looks one of them up (a division and a load) and the others get it by a shuffle
  constexpr int U = 8;
  for (unsigned base = static_cast<unsigned>(rank) * per; base < static_cast<unsigned>(m_end); base += U * ROWS) {
    int found = -1;
    const unsigned at = base + rl + cl * ROWS;
    if (at < static_cast<unsigned>(m_end)) {
      const int m = static_cast<int>(at), b = m / K, k = m - b * K;
      const int slot = (b * E + e) * K + k;              // (B*E*K and B*T fit in 31 bits)
      found = slot;
      if (Ind) {
        const long long t = load_index(Ind, index_dtype, slot);
        if (t >= 0 && t < T_) {
          found = b * T_ + static_cast<int>(t);
        } else {
          found = -1;
          status.report(EGS_STATUS_INDEX_OUT_OF_RANGE);
        }
      }
    }
    long long row[U];
#pragma unroll
    for (int u = 0; u < U; ++u) row[u] = __shfl_sync(0xffffffffu, found, (tid & 24) | u);
    if (VEC) {
      uint4 x[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        x[u] = (row[u] >= 0 && col < N) ? *reinterpret_cast<const uint4*>(Src + row[u] * N + col) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        auto at = [&](int u) { return to_f32<T>(reinterpret_cast<const T*>(&x[u])[i]); };
        add(i, ((at(0) + at(1)) + (at(2) + at(3))) + ((at(4) + at(5)) + (at(6) + at(7))));
      }
    } else {
      float x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] = (row[u] >= 0 && col < N) ? to_f32<T>(Src[row[u] * N + col]) : 0.f;
      add(0, ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7])));
    }
  }
#pragma unroll
  for (int i = 0; i < PER; ++i) part[rl][cl * PER + i] = isfinite(low[i]) ? acc[i] + low[i] : acc[i];      // (infinities leave no rest)
  __syncthreads();
  if (tid < COLS) {
    double s = 0.0;
    for (int r = 0; r < ROWS; ++r) s += part[r][tid];
    total[tid] = s;
  }
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
  if (rank == 0 && tid < COLS && c0 + tid < N) {
    double s = 0.0;
    const uint32_t mine = static_cast<uint32_t>(__cvta_generic_to_shared(&total[tid]));
    for (int r = 0; r < nranks; ++r) {
      uint32_t addr;
      double v;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(mine), "r"(r));
      asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
      s += v;
    }
    out[static_cast<long long>(e) * N + c0 + tid] = from_f32<T>(static_cast<float>(s));
  }
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");   // nobody's shared memory goes before it is read
}

// ------------------------------------------------------------------------------------------------
// zero fill and fp32 -> dtype conversion
//
// Both are bound by memory.  Large buffers are cut into stretches of kStretch (kConvert) vectors a thread with a CTA for each: handed out
// in order as CTAs leave, the stretches in flight lie together, and 1.07 GB are zeroed in 147 us (7.3 TB/s), 128 MB in 24.6 and 64 MB in 14.3; by a
// few waves of CTAs that stride over all of it 176, 26.6 and 16.4 us.  24 MB take those 8.3 us, stretches 9.0.  Where a kernel starts under the
// fill it does so under a grid of few waves only, and the fill in front of a 16-bit scatter has more to do in each CTA: whole scatters of
// 134 MB take 172 us with stretches and 170 without, of 268 MB 107 and 113, of 1.07 GB 1340 and 1367.  From 160 MB on they take 0.93 to 1.01 of the
// time without, 1.02 to 1.03 in front of a long contraction (171 MB, 504 -> 1352 features: 107.6 and 104.8), and 0.93 to 0.99 where a hot row
// doubles the bytes.
// ------------------------------------------------------------------------------------------------
constexpr int kStretch = 4;
constexpr int kConvert = 2;                        // ... and twice as many 16-byte loads
constexpr size_t kManyCtas = 32 << 20, kManyEarly = 160 << 20;     // bytes from which on; where dependents start early
constexpr unsigned kFewCtas = 148 * 8;             // a few waves of the 148 SMs

template <int THREADS>
__device__ __forceinline__ void fill_vectors(uint4* p, size_t n, bool many) {
  const uint4 z = make_uint4(0, 0, 0, 0);
  if (many) {
    for (size_t b = blockIdx.x; b * (THREADS * kStretch) < n; b += gridDim.x)
#pragma unroll
      for (int j = 0; j < kStretch; ++j) {
        const size_t i = b * (THREADS * kStretch) + j * THREADS + threadIdx.x;
        if (i < n) p[i] = z;
      }
  } else {
    const size_t stride = static_cast<size_t>(gridDim.x) * THREADS;
    for (size_t i = static_cast<size_t>(blockIdx.x) * THREADS + threadIdx.x; i < n; i += stride) p[i] = z;
  }
}

__global__ void __launch_bounds__(256) fill_zero_kernel(uint4* p16, size_t n16, unsigned char* tail,
                                                       size_t ntail, int early) {
  pdl_wait();
  if (early) pdl_trigger();
  fill_vectors<256>(p16, n16, gridDim.x > kFewCtas);
  if (blockIdx.x == 0 && threadIdx.x < ntail) tail[threadIdx.x] = 0;
}

__global__ void __launch_bounds__(256) fill_zero_bytes_kernel(unsigned char* p, size_t n, int early) {
  pdl_wait();
  if (early) pdl_trigger();
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) p[i] = 0;
}

// 8 float32 values -> 8 elements of T with vector loads and one 16-byte store (T is a 16-bit type)
template <typename T>
__device__ __forceinline__ void store8(const float4& a, const float4& b, T* dst) {
  T v[8] = {from_f32<T>(a.x), from_f32<T>(a.y), from_f32<T>(a.z), from_f32<T>(a.w),
            from_f32<T>(b.x), from_f32<T>(b.y), from_f32<T>(b.z), from_f32<T>(b.w)};
  *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(v);
}
template <typename T>
__device__ __forceinline__ void convert8(const float* src, T* dst) {
  const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
  store8<T>(a, b, dst);
}

template <typename T>
__global__ void __launch_bounds__(256) convert_from_f32_kernel(const float* src, T* dst,
                                                              size_t n, int early) {
  pdl_wait();
  if (early) pdl_trigger();
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  const size_t i0 = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const bool vec = sizeof(T) == 2 && ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0;
  const size_t n8 = vec ? n / 8 : 0;
  if (gridDim.x > kFewCtas) {
    for (size_t b = blockIdx.x; b * (256 * kConvert) < n8; b += gridDim.x) {
      float4 v[kConvert][2];
#pragma unroll
      for (int j = 0; j < kConvert; ++j) {
        const size_t i = b * (256 * kConvert) + j * 256 + threadIdx.x;
        if (i < n8) {
          v[j][0] = *reinterpret_cast<const float4*>(src + 8 * i);
          v[j][1] = *reinterpret_cast<const float4*>(src + 8 * i + 4);
        }
      }
#pragma unroll
      for (int j = 0; j < kConvert; ++j) {
        const size_t i = b * (256 * kConvert) + j * 256 + threadIdx.x;
        if (i < n8) store8<T>(v[j][0], v[j][1], dst + 8 * i);
      }
    }
  } else {
    for (size_t i = i0; i < n8; i += stride) convert8<T>(src + 8 * i, dst + 8 * i);
  }
  for (size_t i = n8 * 8 + i0; i < n; i += stride) dst[i] = from_f32<T>(src[i]);
}

template <typename T>
__global__ void __launch_bounds__(256) convert_to_f32_kernel(const T* src, float* dst,
                                                            size_t n) {
  pdl_wait();
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
    dst[i] = to_f32<T>(src[i]);
}

// ---- 16-bit scatter: preparation and finish -------------------------------------------------------
// Adding straight into a bf16/fp16 output rounds at every addition, which is accurate enough only while few
// contributions meet in one token row; summing in float32 rows and rounding once is always accurate but costs
// a float32 fill, float32 atomics on a buffer twice the size and a conversion pass.  The choice is made on the
// device, per call, from the actual indices: a plan's kPlanHot selects the float32 rows.  One hot row anywhere selects them for every row
// of the call, so that what a row is summed in does not depend on its own luck alone.
// The ids of a batch element are counted in shared memory by one CTA (4096 ids: about 2 us) of a kernel of their own, with a flag
// per CTA; the kernel that zeroes what the additions go to starts under it (dependent launch) and collects the flags: 2 us of the
// chain.  With a single batch element, or few ids and token rows in all (kPrepOwnIds of each: as long to count as the second launch
// takes; 32712 counters a CTA took a pass with 133 MB of rows from 172 to 218 us), the CTAs of the zeroing kernel count everything themselves: a serving pass of one 64-token prompt has 25 us in all.
// Sequences beyond kPrepCounters tokens share counters (token id modulo kPrepCounters): that can choose the float32 rows where
// they are not needed, never the reverse.
constexpr int kPrepThreads = 512;
constexpr int kPrepCounters = 50 * 1024;
constexpr int kPrepCountCtas = 4 * 148;
constexpr int kPrepOwnIds = 8192;

// whether a token row of batch elements b0 .. b0 + nb - 1 gets more than `limit` contributions, counted by the whole CTA;
// cnt: [min(nb * T_, kPrepCounters)].  Eight ids of a thread are on their way at a time: one after the other, the counting of 8 batch
// elements of 8192 ids took 17 us of device time, all scatters of such sizes 8 us longer (bf16, T=2048, 64 experts, 512 -> 2048 features: 140 us,
// now 132; 32 elements of 4096 ids, 128 -> 512 features: 54 and 50).  Four where the CTAs that fill count for themselves (see
// scatter_prepare_kernel).
template <bool ONE, int kAtOnce>
__device__ __forceinline__ int has_hot_row(const void* ind, int index_dtype, int b0, int nb, int T_, int EK, int limit, int* cnt) {
  const int tid = threadIdx.x, nc = static_cast<int>(min(static_cast<long long>(nb) * T_, static_cast<long long>(kPrepCounters)));
  for (int t = tid; t < nc; t += kPrepThreads) cnt[t] = 0;
  __syncthreads();
  const unsigned ids = ONE ? EK : nb * EK;
  int over = 0;
  for (unsigned s0 = tid; s0 < ids; s0 += kAtOnce * kPrepThreads) {
    long long id[kAtOnce];
#pragma unroll
    for (int i = 0; i < kAtOnce; ++i) {
      const unsigned s = s0 + i * kPrepThreads;
      id[i] = s < ids ? load_index(ind, index_dtype, static_cast<long long>(b0) * EK + s) : -1;
    }
#pragma unroll
    for (int i = 0; i < kAtOnce; ++i) {
      if (id[i] < 0 || id[i] >= T_) continue;
      int at = static_cast<int>(id[i]) + (ONE ? 0 : static_cast<int>((s0 + i * kPrepThreads) / static_cast<unsigned>(EK)) * T_);
      if (at >= nc) at %= nc;
      over |= atomicAdd(&cnt[at], 1) >= limit;
    }
  }
  return __syncthreads_or(over);         // (and the counters may be used again)
}

__global__ void __launch_bounds__(kPrepThreads) scatter_count_kernel(const void* ind, int index_dtype, int B, int T_, int EK,
                                                                     int limit, int* flags) {
  extern __shared__ int prep_cnt[];
  pdl_wait();
  pdl_trigger();
  int flag = 0;
  for (int b = blockIdx.x; b < B && !flag; b += gridDim.x) flag = has_hot_row<true, 8>(ind, index_dtype, b, 1, T_, EK, limit, prep_cnt);
  if (threadIdx.x == 0) flags[blockIdx.x] = flag;
}

// COUNT: the CTAs count for themselves, an instance of its own.  Four CTAs of either are on an SM, as many as the grid counts on: with eight ids at a
// time counting took registers for three, and the fourth quarter of the grid counted when the others had filled (bf16, whole scatters: 2
// batch elements of 1956 tokens, 156 ids each, 120 -> 928 features 9.9 us without, 11.0 with eight ids, 10.0 with four; 1 of 5006, 448 ids, 480 -> 1632
// 13.5, 14.4 and 13.3; 1 of 8192, 8192 ids, 256 -> 1024 26.3, 20.3 and 19.7).
template <typename T, bool COUNT>
__global__ void __launch_bounds__(kPrepThreads, 4) scatter_prepare_kernel(const void* ind, int index_dtype, int B, int T_, int EK,
                                                                       const int* info, const int* flags, int nflags,
                                                                       int limit, int* plan, float* acc,
                                                                       T* out, size_t n, int zero_output, StatusRef status) {
  extern __shared__ int prep_cnt[];      // without `info` and `flags`
  if (nflags > 0) pdl_trigger();         // (the counting kernel has waited: the scatter may begin under it)
  pdl_wait();
  if (nflags == 0) pdl_trigger();
  const int tid = threadIdx.x;
  int flag = 0;
  if (info) {
    flag = info[0] > limit;
    if (info[2] && blockIdx.x == 0 && tid == 0) status.report(EGS_STATUS_INDEX_OUT_OF_RANGE);
  } else if (nflags > 0) {
    for (int i = tid; i < nflags; i += kPrepThreads) flag |= flags[i];
    flag = __syncthreads_or(flag);
  } else if (COUNT) {
    flag = B == 1 ? has_hot_row<true, 4>(ind, index_dtype, 0, 1, T_, EK, limit, prep_cnt) : has_hot_row<false, 4>(ind, index_dtype, 0, B, T_, EK, limit, prep_cnt);
  }
  if (blockIdx.x == 0 && tid < kPlanWords) plan[tid] = tid == kPlanHot ? flag : 0;
  // (n is a multiple of 8 elements and both buffers are 16-byte aligned: tensor-core path only)
  if (zero_output) {
    fill_vectors<kPrepThreads>(flag ? reinterpret_cast<uint4*>(acc) : reinterpret_cast<uint4*>(out), flag ? n / 4 : n / 8, gridDim.x > kFewCtas);
  } else if (flag) {                     // seed the float32 rows with what the output holds
    const size_t stride = static_cast<size_t>(gridDim.x) * kPrepThreads;
    for (size_t i = static_cast<size_t>(blockIdx.x) * kPrepThreads + tid; i < n; i += stride) acc[i] = to_f32<T>(out[i]);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) scatter_finish_kernel(const int* plan, const float* acc,
                                                            T* out, size_t n) {
  pdl_wait();
  pdl_trigger();
  if (!*plan) return;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n / 8; i += stride) convert8<T>(acc + 8 * i, out + 8 * i);
}

int grid_for(size_t work_items, int per_block, bool many = false) {
  size_t blocks = (work_items + per_block - 1) / per_block;
  if (blocks > kFewCtas && !many) blocks = kFewCtas;
  if (blocks < 1) blocks = 1;
  return static_cast<int>(blocks);
}

}  // namespace

// Tile width over n features in units of 32, at most `most`: the least padding, the widest of equals.  The widest of all where a
// narrower tile's columns would not fit in a grid's y (65535 blocks).
static int width_in_32s(int n, int most) {
  int best = most, best_pad = 1 << 30;
  for (int w = 1; w <= most; ++w) {
    const int tile = 32 * w, tiles = (n + tile - 1) / tile, pad = tiles * tile - n;
    if (pad <= best_pad && tiles <= 65535) {
      best = w;
      best_pad = pad;
    }
  }
  return best;
}

cudaError_t launch_generic_rowgemm(const RowGemmParams& p, bool scatter, int dtype, cudaStream_t st) {
  const int nj = width_in_32s(p.N, 4);
  dim3 grid((p.M + TM - 1) / TM, (p.N + 32 * nj - 1) / (32 * nj), p.E);
  cudaError_t err;
#define EGS_LAUNCH_NJ(TY, NJV, CTAS)                                                       \
  do {                                                                                     \
    if (scatter) err = launch_kernel(generic_rowgemm_kernel<TY, true, NJV, CTAS>, grid, NTHREADS, 0, st, true, p);      \
    else err = launch_kernel(generic_rowgemm_kernel<TY, false, NJV, CTAS>, grid, NTHREADS, 0, st, true, p);             \
  } while (0)
#define EGS_LAUNCH(TY)                       \
  do {                                       \
    if (nj == 1) EGS_LAUNCH_NJ(TY, 1, 4);    \
    else if (nj == 2) EGS_LAUNCH_NJ(TY, 2, 4);  \
    else if (nj == 3 && p.C <= TK) EGS_LAUNCH_NJ(TY, 3, 4);  \
    else if (nj == 3) EGS_LAUNCH_NJ(TY, 3, 3);  \
    else EGS_LAUNCH_NJ(TY, 4, 3);            \
  } while (0)
  if (dtype == EGS_F32) EGS_LAUNCH(float);
  else if (dtype == EGS_F16) EGS_LAUNCH(__half);
  else EGS_LAUNCH(__nv_bfloat16);
#undef EGS_LAUNCH
#undef EGS_LAUNCH_NJ
  count_launch();
  return err;
}

// Tile over FG x FD and the split of the contraction: about four CTAs per SM (eight of 64 threads with small tiles: 108000 rows 7 x 110 54 -> 42 us,
// but 81 -> 89 at 101 x 101), and no fewer than 64 rows in a range, below which adding the partial tile costs more than multiplying it.
void configure_generic_dweight(DWeightParams& p) {
  p.row_tiles = width_in_32s(p.FG, 4);
  p.BN = 32 * width_in_32s(p.FD, 2);
  const long long tiles = static_cast<long long>((p.FG + 32 * p.row_tiles - 1) / (32 * p.row_tiles)) * ((p.FD + p.BN - 1) / p.BN) * p.E;
  const long long ctas = p.BN > 32 && p.row_tiles <= 2 ? 8 * 148 : 4 * 148;
  long long want = (ctas + tiles - 1) / tiles;
  const long long most = (p.M + 63) / 64;
  if (want > most) want = most;
  if (want < 1) want = 1;
  long long rows = (p.M + want - 1) / want;
  rows = (rows + TK - 1) / TK * TK;
  p.rows_per_split = static_cast<int>(rows);
  p.splits = static_cast<int>((p.M + rows - 1) / rows);
}

template <typename T, int FI>
static cudaError_t launch_dweight(const DWeightParams& p, cudaStream_t st) {
  const dim3 grid((p.FG + 32 * FI - 1) / (32 * FI), (p.FD + p.BN - 1) / p.BN, p.E * p.splits);
  if (p.BN == 32) return launch_kernel(generic_dweight_kernel<T, FI, 1>, grid, NTHREADS, 0, st, true, p);
  if constexpr (sizeof(T) == 4) {        // see generic_dweight_wide_kernel
    if (static_cast<long long>(grid.x) * grid.y * grid.z < 2 * 148) return launch_kernel(generic_dweight_kernel<T, FI, 2>, grid, NTHREADS, 0, st, true, p);
  }
  return launch_kernel(generic_dweight_wide_kernel<T, FI, 2>, grid, kWideThreads, 0, st, true, p);
}
template <typename T>
static cudaError_t launch_dweight(const DWeightParams& p, cudaStream_t st) {
  return p.row_tiles == 1 ? launch_dweight<T, 1>(p, st) : p.row_tiles == 2 ? launch_dweight<T, 2>(p, st) : p.row_tiles == 3 ? launch_dweight<T, 3>(p, st) : launch_dweight<T, 4>(p, st);
}

cudaError_t launch_generic_dweight(const DWeightParams& p, int dtype, cudaStream_t st) {
  const cudaError_t err = dtype == EGS_F32 ? launch_dweight<float>(p, st) : dtype == EGS_F16 ? launch_dweight<__half>(p, st) : launch_dweight<__nv_bfloat16>(p, st);
  count_launch();
  return err;
}

template <typename T, bool VEC>
static cudaError_t launch_row_sum(const void* Src, const void* Ind, int index_dtype, void* out, int B, int T_, int E, int K, int N,
                                  StatusRef status, cudaStream_t st) {
  constexpr int cols = 8 * (VEC ? 16 / static_cast<int>(sizeof(T)) : 1);
  const int M = B * K, blocks = (N + cols - 1) / cols;
  // CTAs per cluster: up to eight per SM in all (they are latency chains: id, row, sum), at least 128 rows each
  int ranks = 1;
  while (ranks < 8 && static_cast<long long>(blocks) * E * ranks < 8 * 148 && M >= 128 * 2 * ranks) ranks *= 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ranks * blocks, E);
  cfg.blockDim = dim3(kSumThreads);
  cfg.stream = st;
  // (not a dependent launch: its CTAs, several to an SM, would gather on the SMs that the kernel before it leaves first and stay there:
  // 33 us of row sums then took 48)
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = ranks;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, expert_row_sum_kernel<T, VEC>, static_cast<const T*>(Src), Ind, index_dtype, static_cast<T*>(out), T_, E, K,
                            N, M, ranks, status);
}

cudaError_t launch_expert_row_sum(const void* Src, const void* Ind, int index_dtype, void* out, int B, int T, int E, int K, int N,
                                  int dtype, StatusRef status, cudaStream_t st) {
  const bool vec = (reinterpret_cast<uintptr_t>(Src) & 15u) == 0 && (N * (dtype == EGS_F32 ? 4ll : 2ll)) % 16 == 0;
  cudaError_t err;
#define EGS_SUM(TY) \
  err = vec ? launch_row_sum<TY, true>(Src, Ind, index_dtype, out, B, T, E, K, N, status, st) : launch_row_sum<TY, false>(Src, Ind, index_dtype, out, B, T, E, K, N, status, st)
  if (dtype == EGS_F32) EGS_SUM(float);
  else if (dtype == EGS_F16) EGS_SUM(__half);
  else EGS_SUM(__nv_bfloat16);
#undef EGS_SUM
  count_launch();
  return err;
}

cudaError_t launch_fill_zero(void* ptr, size_t bytes, cudaStream_t st, bool early) {
  if (bytes == 0) return cudaSuccess;
  const uintptr_t a = reinterpret_cast<uintptr_t>(ptr);
  cudaError_t err;
  if (a % 16 != 0) {
    err = launch_kernel(fill_zero_bytes_kernel, grid_for(bytes, 256), 256, 0, st, true, static_cast<unsigned char*>(ptr), bytes, early ? 1 : 0);
  } else {
    const size_t n16 = bytes / 16, ntail = bytes % 16;
    err = launch_kernel(fill_zero_kernel, grid_for(n16, 256 * kStretch, bytes > (early ? kManyEarly : kManyCtas)), 256, 0, st, true, static_cast<uint4*>(ptr), n16,
                        static_cast<unsigned char*>(ptr) + n16 * 16, ntail, early ? 1 : 0);
  }
  count_launch();
  return err;
}

cudaError_t launch_convert_from_f32(const float* src, void* dst, size_t n, int dtype, cudaStream_t st, bool early) {
  if (n == 0) return cudaSuccess;
  const int grid = n * sizeof(float) > kManyCtas ? grid_for(n, 8 * 256 * kConvert, true) : grid_for(n, 256 * 4);
  cudaError_t err;
  if (dtype == EGS_F16) err = launch_kernel(convert_from_f32_kernel<__half>, grid, 256, 0, st, true, src, static_cast<__half*>(dst), n, early ? 1 : 0);
  else if (dtype == EGS_BF16)
    err = launch_kernel(convert_from_f32_kernel<__nv_bfloat16>, grid, 256, 0, st, true, src, static_cast<__nv_bfloat16*>(dst), n, early ? 1 : 0);
  else return cudaErrorInvalidValue;
  count_launch();
  return err;
}

template <typename T>
static cudaError_t prepare(const void* Ind, int index_dtype, int B, int T_, int EK, const int* info, int limit, int* flags, int* plan,
                           float* acc, void* out16, size_t n, int zero_output, StatusRef status, cudaStream_t st) {
  const bool count = info == nullptr && EK > limit;
  const long long ids = static_cast<long long>(B) * EK, rows = static_cast<long long>(B) * T_;
  const bool own_count = count && (B == 1 || (ids <= kPrepOwnIds && rows <= kPrepOwnIds));
  const long long counters = own_count ? rows : T_;
  const size_t smem = count ? static_cast<size_t>(counters < kPrepCounters ? counters : kPrepCounters) * sizeof(int) : 0;
  cudaError_t err = cudaSuccess;
  int nflags = 0;
  if (count && !own_count) {
    nflags = B < kPrepCountCtas ? B : kPrepCountCtas;
    if (smem > 48 * 1024) err = ensure_smem_optin<scatter_count_kernel>(kPrepCounters * static_cast<int>(sizeof(int)));
    if (err != cudaSuccess) return err;
    err = launch_kernel(scatter_count_kernel, nflags, kPrepThreads, smem, st, true, Ind, index_dtype, B, T_, EK, limit, flags);
    count_launch();
    if (err != cudaSuccess) return err;
  }
  // four CTAs per SM, or as many as there are stretches; each with at least 4 KB to zero and, where it counts, no more ids than half the
  // elements it zeroes
  size_t grid = 4 * 148;
  if (zero_output && n * sizeof(T) > kManyEarly && !own_count) grid = (n / 8 + kPrepThreads * kStretch - 1) / (kPrepThreads * kStretch);
  const size_t by_bytes = n * sizeof(T) / 4096, by_count = own_count ? n / (2 * static_cast<size_t>(ids)) : grid;
  if (grid > by_bytes) grid = by_bytes;
  if (grid > by_count) grid = by_count;
  if (grid < 1) grid = 1;
  if (own_count && smem > 48 * 1024) err = ensure_smem_optin<scatter_prepare_kernel<T, true>>(kPrepCounters * static_cast<int>(sizeof(int)));
  if (err != cudaSuccess) return err;
  err = launch_kernel(own_count ? scatter_prepare_kernel<T, true> : scatter_prepare_kernel<T, false>, static_cast<unsigned>(grid), kPrepThreads,
                      own_count ? smem : 0, st, true, Ind, index_dtype, B, T_, EK, info, flags, nflags, limit, plan, acc, static_cast<T*>(out16), n,
                      zero_output, status);
  count_launch();
  return err;
}

cudaError_t launch_scatter_prepare(const void* Ind, int index_dtype, int B, int T, int E, int K, const int* csr_info, int limit, int* flags,
                                   int* plan, float* acc, void* out16, int N, int zero_output, int dtype, StatusRef status, cudaStream_t st) {
  const size_t n = static_cast<size_t>(B) * T * N;
  if (n == 0) return cudaSuccess;
  const int ek = E * K;      // B*E*K fits in 32 bits
  if (dtype == EGS_F16) return prepare<__half>(Ind, index_dtype, B, T, ek, csr_info, limit, flags, plan, acc, out16, n, zero_output, status, st);
  if (dtype == EGS_BF16)
    return prepare<__nv_bfloat16>(Ind, index_dtype, B, T, ek, csr_info, limit, flags, plan, acc, out16, n, zero_output, status, st);
  return cudaErrorInvalidValue;
}

cudaError_t launch_scatter_finish(const int* plan, const float* acc, void* out16, size_t n, int dtype, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const int grid = grid_for(n, 256 * 8 * 4);             // a few waves of CTAs: mostly they find nothing to do
  cudaError_t err;
  if (dtype == EGS_F16) err = launch_kernel(scatter_finish_kernel<__half>, grid, 256, 0, st, true, plan, acc, static_cast<__half*>(out16), n);
  else if (dtype == EGS_BF16)
    err = launch_kernel(scatter_finish_kernel<__nv_bfloat16>, grid, 256, 0, st, true, plan, acc, static_cast<__nv_bfloat16*>(out16), n);
  else return cudaErrorInvalidValue;
  count_launch();
  return err;
}

cudaError_t launch_convert_to_f32(const void* src, float* dst, size_t n, int dtype, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const int grid = grid_for(n, 256 * 4);
  cudaError_t err;
  if (dtype == EGS_F16) err = launch_kernel(convert_to_f32_kernel<__half>, grid, 256, 0, st, true, static_cast<const __half*>(src), dst, n);
  else if (dtype == EGS_BF16)
    err = launch_kernel(convert_to_f32_kernel<__nv_bfloat16>, grid, 256, 0, st, true, static_cast<const __nv_bfloat16*>(src), dst, n);
  else return cudaErrorInvalidValue;
  count_launch();
  return err;
}

}  // namespace egs

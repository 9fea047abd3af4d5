// Router-side index preparation and its consumers (sm_100a build, no tensor-core code: integer and byte work).
//
// The path's index tensor Ind[B,E,K] ("for batch element b, expert e processes tokens Ind[b,e,:]", reference README.md:7)
// is produced by a router in front of the gather and consumed token-major by the scatter.  The reference has neither
// step (its tests draw Ind with torch.randint, test_all.py:16, and its scatter resolves collisions with atomics,
// egs/triton_kernels.py:235-247).  Here:
//   route_topk      expert-choice routing: Ind[b,e,:] = the K tokens with the highest score[b,:,e], best first
//                   (radix select over the order-preserving bit pattern of the scores, then a bitonic sort of the K)
//   csr_*           token-major CSR of Ind by counting sort: counts / offsets per token row (b,t) and the slot ids
//                   routed to it in ascending order; also the heaviest row, the number of rows touched and a flag for
//                   out-of-range ids.  One build per step serves both scatters of the step and the 16-bit scatter's
//                   choice between direct 16-bit additions and float32 rows.
//   compact_index   Ind -> int32 / int16 with a range check
//   csr_scatter     operator S evaluated token-major from the CSR: every token row is owned by one CTA, which sums its
//                   contributions in a fixed order and STORES the row (zeros for untouched rows): no atomics, no zero
//                   fill, bit-reproducible.  It re-reads W[e] for every contribution, so it only pays where the
//                   contraction is small; the expert-major tensor-core kernels remain the fast path.
#include "egs_internal.cuh"

namespace egs {

namespace {

// ---- order-preserving key of a float: larger float <=> larger unsigned key ----
__device__ __forceinline__ uint32_t float_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// ---- route_topk, keys in registers ---------------------------------------------------------------------------------------
// A CTA serves EG neighbouring experts of one batch element, WPE warps each.  The [T, EG] block of scores is read in whole
// sectors (the experts are the contiguous direction: one expert alone would fetch eight times its bytes) and turned through
// shared memory so that every thread ends up with R keys of its expert in registers.  The K-th largest key is then built bit
// by bit - R compares and a reduction per bit - and the search stops as soon as exactly K keys lie at or above the candidate,
// after about 20 of 32 bits for scores without ties.  What bounds it is that chain of reductions and, before it, of chunks read one
// after the other, not the bytes: few (batch, expert) pairs get more warps each (see launch_route_topk).
// B=32, T=2048, E=64, K=128: 28 us; 127 us with one CTA per expert column and shared-memory histograms.
constexpr int kSelChunk = 8;          // keys per thread and chunk of the turn through shared memory
constexpr int kSelMaxKeys = 64;       // keys per thread

template <int WPE>
__device__ __forceinline__ void expert_sync(int eg) {
  if (WPE == 1) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(eg + 1), "r"(WPE * 32) : "memory");
}
// sum over the expert's threads; red: two sets of WPE slots of this expert, used in turn (par), so that one barrier is enough
template <int WPE>
__device__ __forceinline__ unsigned expert_sum(unsigned v, unsigned* red, int par, int eg, int w, int lane) {
  v = __reduce_add_sync(0xffffffffu, v);
  if (WPE == 1) return v;
  red += (par & 1) * WPE;
  if (lane == 0) red[w] = v;
  expert_sync<WPE>(eg);
  v = 0;
#pragma unroll
  for (int i = 0; i < WPE; ++i) v += red[i];
  return v;
}

template <int WPE, int R>
__global__ void __launch_bounds__(512) route_topk_regs_kernel(const float* scores, void* ind, int index_dtype,
                                                              int T, int E, int K, int eg_log2, int P) {
  constexpr int CT = WPE * 32 * kSelChunk;   // tokens per chunk
  extern __shared__ __align__(16) unsigned char sel_smem[];
  __shared__ unsigned red_s[32], count_s[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int eg = warp / WPE, w = warp - eg * WPE;       // expert within the CTA, warp within the expert
  const int EG = 1 << eg_log2;
  const int pitch = CT + 4;                             // words; neighbouring experts 4 banks apart
  uint32_t* turn = reinterpret_cast<uint32_t*>(sel_smem);                       // [EG][pitch], later the lists
  unsigned long long* sel = reinterpret_cast<unsigned long long*>(sel_smem) + static_cast<size_t>(eg) * P;
  const int groups = (E + EG - 1) / EG;
  const int b = blockIdx.x / groups, e0 = (blockIdx.x - b * groups) * EG;
  const float* base = scores + static_cast<long long>(b) * T * E + e0;
  const int nthreads = EG * WPE * 32;

  pdl_wait();
  pdl_trigger();
  uint32_t key[R];
  float v[kSelChunk];
  auto fetch = [&](int t0) {
#pragma unroll
    for (int i = 0; i < kSelChunk; ++i) {
      const int idx = tid + i * nthreads, t = t0 + (idx >> eg_log2), g = idx & (EG - 1);
      v[i] = (t < T && e0 + g < E) ? base[static_cast<long long>(t) * E + g] : 0.f;
    }
  };
  fetch(0);
#pragma unroll
  for (int c = 0; c < R / kSelChunk; ++c) {
    if (c * CT < T) {                                   // (uniform over the CTA)
#pragma unroll
      for (int i = 0; i < kSelChunk; ++i) {
        const int idx = tid + i * nthreads;
        turn[(idx & (EG - 1)) * pitch + (idx >> eg_log2)] = float_key(v[i]);
      }
      __syncthreads();
      if ((c + 1) * CT < T) fetch((c + 1) * CT);
    }
#pragma unroll
    for (int i = 0; i < kSelChunk; ++i) {
      const int tl = i * (WPE * 32) + w * 32 + lane;
      key[c * kSelChunk + i] = (c * CT + tl < T) ? turn[eg * pitch + tl] : 0u;      // 0: below every candidate
    }
    if (c * CT < T) __syncthreads();
  }
  if (e0 + eg >= E) return;       // no CTA-wide barrier below

  unsigned* red = red_s + eg * 2 * WPE;
  uint32_t th = 0;
  bool exact = false;             // exactly K keys are >= th
  for (int bit = 31; bit >= 0 && !exact; --bit) {
    const uint32_t cand = th | (1u << bit);
    unsigned n = 0;
#pragma unroll
    for (int i = 0; i < R; ++i) n += (key[i] >= cand) ? 1u : 0u;
    n = expert_sum<WPE>(n, red, bit, eg, w, lane);
    if (n >= static_cast<unsigned>(K)) th = cand;
    exact = n == static_cast<unsigned>(K);
  }
  // collect all keys above the threshold (at it, too, when they are exactly K), in any order: a thread's keys go to consecutive
  // places, behind those of the lanes before it and of the warps that got there first
  const uint32_t from = exact ? th : th + 1u;            // th is the largest key only if exact or tied at it: no wrap matters
  const bool all_ones = !exact && th == 0xFFFFFFFFu;
  if (w == 0 && lane == 0) count_s[eg] = 0;
  expert_sync<WPE>(eg);
  unsigned mine = 0;
#pragma unroll
  for (int i = 0; i < R; ++i) mine += (key[i] >= from) ? 1u : 0u;
  if (all_ones) mine = 0;
  unsigned incl = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += o;
  }
  unsigned pos = 0;
  if (lane == 31) pos = atomicAdd(&count_s[eg], incl);
  pos = __shfl_sync(0xffffffffu, pos, 31) + incl - mine;
  if (mine) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (key[i] >= from) {
        const int t = (i / kSelChunk) * CT + (i % kSelChunk) * (WPE * 32) + w * 32 + lane;
        sel[pos++] = (static_cast<unsigned long long>(key[i]) << 32) | (0xFFFFFFFFu - static_cast<unsigned>(t));
      }
    }
  }
  expert_sync<WPE>(eg);
  if (!exact) {
    // keys equal to the K-th: the lowest token ids fill the list (tokens ascend with the register index, then with the thread)
    unsigned n_gt = count_s[eg];
    for (int i = 0; i < R && n_gt < static_cast<unsigned>(K); ++i) {
      uint32_t k = 0;
#pragma unroll
      for (int j = 0; j < R; ++j)
        if (j == i) k = key[j];
      const int t = (i / kSelChunk) * CT + (i % kSelChunk) * (WPE * 32) + w * 32 + lane;
      const bool eq = t < T && k == th;
      const unsigned m = __ballot_sync(0xffffffffu, eq);
      unsigned before = __popc(m & ((1u << lane) - 1u)), total = __popc(m);
      if (WPE > 1) {
        expert_sync<WPE>(eg);
        if (lane == 0) red[w] = __popc(m);
        expert_sync<WPE>(eg);
        total = 0;
#pragma unroll
        for (int j = 0; j < WPE; ++j) {
          if (j < w) before += red[j];
          total += red[j];
        }
      }
      if (eq && n_gt + before < static_cast<unsigned>(K))
        sel[n_gt + before] = (static_cast<unsigned long long>(k) << 32) | (0xFFFFFFFFu - static_cast<unsigned>(t));
      n_gt += total;
    }
  }
  // bitonic sort of the K selected (padded to a power of two with zeros, which sort last), descending
  const int me = w * 32 + lane;
  for (int i = K + me; i < P; i += WPE * 32) sel[i] = 0ull;
  expert_sync<WPE>(eg);
  for (int size = 2; size <= P; size <<= 1)
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = me; i < P / 2; i += WPE * 32) {
        const int lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
        const unsigned long long x = sel[lo], y = sel[hi];
        if ((x < y) == ((lo & size) == 0)) { sel[lo] = y; sel[hi] = x; }
      }
      expert_sync<WPE>(eg);
    }
  const long long out0 = (static_cast<long long>(b) * E + e0 + eg) * K;
  for (int k = me; k < K; k += WPE * 32) {
    const long long tok = static_cast<long long>(0xFFFFFFFFu - static_cast<unsigned>(sel[k] & 0xFFFFFFFFull));
    if (index_dtype == EGS_I64) static_cast<long long*>(ind)[out0 + k] = tok;
    else if (index_dtype == EGS_I32) static_cast<int*>(ind)[out0 + k] = static_cast<int>(tok);
    else static_cast<short*>(ind)[out0 + k] = static_cast<short>(tok);
  }
}

// ---- route_topk for sequences beyond the registers -----------------------------------------------------------------------
constexpr int kTopkThreads = 256;
constexpr int kTopkMaxK = 1024;

// One CTA per (b, e).  scores: [B, T, E] float32.  Ties are broken towards the lower token id.  NaN scores order above
// +inf (their bit pattern), i.e. they are selected first.
__global__ void __launch_bounds__(kTopkThreads) route_topk_kernel(const float* __restrict__ scores, void* __restrict__ ind,
                                                                  int index_dtype, int B, int T, int E, int K) {
  __shared__ unsigned hist[256];
  __shared__ unsigned s_prefix, s_remaining, s_count_gt, s_count_eq;
  __shared__ unsigned long long sel[kTopkMaxK];    // (key << 32) | (0xFFFFFFFF - token): descending order = best first, low token first
  const int b = blockIdx.x / E, e = blockIdx.x - b * E;
  const float* col = scores + (static_cast<long long>(b) * T) * E + e;
  const int tid = threadIdx.x;

  // radix select, most significant byte first: after the loop `prefix` is the key of the K-th best element
  unsigned prefix = 0, remaining = static_cast<unsigned>(K);
  for (int shift = 24; shift >= 0; shift -= 8) {
    hist[tid] = 0;
    __syncthreads();
    const unsigned mask = (shift == 24) ? 0u : (0xFFFFFFFFu << (shift + 8));
    for (int t = tid; t < T; t += kTopkThreads) {
      const unsigned key = float_key(col[static_cast<long long>(t) * E]);
      if ((key & mask) == (prefix & mask)) atomicAdd(&hist[(key >> shift) & 255u], 1u);
    }
    __syncthreads();
    if (tid == 0) {
      unsigned need = remaining, bin = 255;
      for (;; --bin) {                       // walk from the largest digit down until the K-th element's bin
        if (hist[bin] >= need || bin == 0) break;
        need -= hist[bin];
      }
      s_prefix = prefix | (bin << shift);
      s_remaining = need;
    }
    __syncthreads();
    prefix = s_prefix;
    remaining = s_remaining;
    __syncthreads();
  }
  // collect: every key above the threshold, plus `remaining` keys equal to it, lowest token ids first
  if (tid == 0) { s_count_gt = 0; s_count_eq = 0; }
  __syncthreads();
  const unsigned n_gt = static_cast<unsigned>(K) - remaining;
  for (int t0 = 0; t0 < T; t0 += kTopkThreads) {          // in token order, so that ties resolve deterministically
    const int t = t0 + tid;
    unsigned key = 0;
    bool gt = false, eq = false;
    if (t < T) {
      key = float_key(col[static_cast<long long>(t) * E]);
      gt = key > prefix;
      eq = key == prefix;
    }
    // rank of this thread among the `eq` threads of this pass (block-wide, by thread index)
    const unsigned ballot_eq = __ballot_sync(0xffffffffu, eq);
    __shared__ unsigned warp_eq[kTopkThreads / 32];
    if ((tid & 31) == 0) warp_eq[tid >> 5] = __popc(ballot_eq);
    __syncthreads();
    unsigned before = s_count_eq;
    for (int w = 0; w < (tid >> 5); ++w) before += warp_eq[w];
    before += __popc(ballot_eq & ((1u << (tid & 31)) - 1u));
    if (gt) {
      const unsigned pos = atomicAdd(&s_count_gt, 1u);
      sel[pos] = (static_cast<unsigned long long>(key) << 32) | (0xFFFFFFFFu - static_cast<unsigned>(t));
    } else if (eq && before < remaining) {
      sel[n_gt + before] = (static_cast<unsigned long long>(key) << 32) | (0xFFFFFFFFu - static_cast<unsigned>(t));
    }
    __syncthreads();
    if (tid == 0) {
      unsigned tot = 0;
      for (int w = 0; w < kTopkThreads / 32; ++w) tot += warp_eq[w];
      s_count_eq += tot;
    }
    __syncthreads();
  }
  // bitonic sort of the K selected (padded to a power of two with zeros, which sort last), descending
  int P = 1;
  while (P < K) P <<= 1;
  for (int i = K + tid; i < P; i += kTopkThreads) sel[i] = 0ull;
  __syncthreads();
  for (int size = 2; size <= P; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = tid; i < P / 2; i += kTopkThreads) {
        const int lo = 2 * i - (i & (stride - 1));
        const int hi = lo + stride;
        const bool desc = ((lo & size) == 0);
        const unsigned long long a = sel[lo], c = sel[hi];
        if ((a < c) == desc) { sel[lo] = c; sel[hi] = a; }
      }
      __syncthreads();
    }
  }
  const long long out0 = (static_cast<long long>(b) * E + e) * K;
  for (int k = tid; k < K; k += kTopkThreads) {
    const long long tok = static_cast<long long>(0xFFFFFFFFu - static_cast<unsigned>(sel[k] & 0xFFFFFFFFull));
    if (index_dtype == EGS_I64) static_cast<long long*>(ind)[out0 + k] = tok;
    else if (index_dtype == EGS_I32) static_cast<int*>(ind)[out0 + k] = static_cast<int>(tok);
    else static_cast<short*>(ind)[out0 + k] = static_cast<short>(tok);
  }
}

// ---- CSR by counting sort, one CTA per batch element ----------------------------------------------------------------------
// A batch element's token rows and slots fit in shared memory for ordinary sizes: counting, the scan and the placement then need
// no global atomics, and two launches do what the general path below does in nine.  The first counts; the second knows how many
// valid slots the batch elements before its own have and places the entries.  Slots of one row come out in ascending order: an
// entry's place is the number of smaller slots in its row (counted among the row's own entries, which are few; every entry is
// ranked by a thread of its own, so a heavy row does not serialise).
// B=32, T=2048, E=64, K=128: nine launches, 38 us of kernels.
constexpr int kCsrBatchThreads = 1024;

// sums over the CTA's threads, every thread gets the totals; red: 32 entries
__device__ __forceinline__ int cta_sum(int v, int* red) {
  v = __reduce_add_sync(0xffffffffu, v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  int s = red[threadIdx.x & 31];
  return __reduce_add_sync(0xffffffffu, s);
}

__global__ void __launch_bounds__(kCsrBatchThreads) csr_batch_count_kernel(const void* ind, int index_dtype, int T, int EK,
                                                                           int* counts, int4* partial) {
  extern __shared__ int cnt[];          // [T]
  __shared__ int red[32];
  const int b = blockIdx.x, tid = threadIdx.x;
  for (int t = tid; t < T; t += kCsrBatchThreads) cnt[t] = 0;
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  int valid = 0, bad = 0;
  for (int s = tid; s < EK; s += kCsrBatchThreads) {
    const long long t = load_index(ind, index_dtype, static_cast<long long>(b) * EK + s);
    if (t >= 0 && t < T) {
      atomicAdd(&cnt[t], 1);
      ++valid;
    } else {
      bad = 1;
    }
  }
  __syncthreads();
  int most = 0, rows = 0;
  for (int t = tid; t < T; t += kCsrBatchThreads) {
    const int c = cnt[t];
    counts[static_cast<long long>(b) * T + t] = c;
    most = max(most, c);
    rows += c > 0;
  }
  valid = cta_sum(valid, red);
  rows = cta_sum(rows, red);
  bad = __syncthreads_or(bad);
  most = __reduce_max_sync(0xffffffffu, most);
  if ((tid & 31) == 0) red[tid >> 5] = most;
  __syncthreads();
  if (tid == 0) {
    for (int i = 0; i < 32; ++i) most = max(most, red[i]);
    partial[b] = make_int4(most, rows, bad ? 1 : 0, valid);
  }
}

__global__ void __launch_bounds__(kCsrBatchThreads) csr_batch_place_kernel(const void* ind, int index_dtype, int T, int EK,
                                                                           const int* counts, const int4* partial,
                                                                           int* offsets, int* entries,
                                                                           int* info) {
  extern __shared__ int csr_smem[];
  __shared__ int red[32];
  int* start = csr_smem;                // [T + 1] first entry of every row, local
  int* cursor = csr_smem + T + 1;       // [T]
  int* list = cursor + T;               // [EK] slots grouped by row, unordered inside a row
  const int b = blockIdx.x, nb = gridDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  pdl_wait();
  pdl_trigger();
  int before = 0;
  for (int i = tid; i < b; i += kCsrBatchThreads) before += partial[i].w;
  before = cta_sum(before, red);
  if (b == 0 && warp == 0) {            // the summary over all batch elements
    int most = 0, rows = 0, bad = 0, valid = 0;
    for (int i = lane; i < nb; i += 32) {
      const int4 q = partial[i];
      most = max(most, q.x);
      rows += q.y;
      bad |= q.z;
      valid += q.w;
    }
    most = __reduce_max_sync(0xffffffffu, most);
    rows = __reduce_add_sync(0xffffffffu, rows);
    bad = __reduce_or_sync(0xffffffffu, bad);
    valid = __reduce_add_sync(0xffffffffu, valid);
    if (lane == 0) {
      info[0] = most;
      info[1] = rows;
      info[2] = bad;
      info[3] = valid;
    }
  }
  // exclusive scan of the counts: a contiguous run of rows per thread, then a scan of the threads' sums
  const int per = (T + kCsrBatchThreads - 1) / kCsrBatchThreads, t0 = min(T, tid * per), t1 = min(T, t0 + per);
  const int* row_counts = counts + static_cast<long long>(b) * T;
  for (int t = tid; t < T; t += kCsrBatchThreads) cursor[t] = row_counts[t];
  __syncthreads();
  int sum = 0;
  for (int t = t0; t < t1; ++t) sum += cursor[t];
  int incl = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += o;
  }
  __syncthreads();
  if (lane == 31) red[warp] = incl;
  __syncthreads();
  int wsum = red[lane];
  const int mine = wsum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, wsum, d);
    if (lane >= d) wsum += o;
  }
  const int wbase = __shfl_sync(0xffffffffu, wsum - mine, warp);
  const int total = __shfl_sync(0xffffffffu, wsum, 31);
  int run = wbase + incl - sum;
  for (int t = t0; t < t1; ++t) {
    const int c = cursor[t];
    start[t] = run;
    cursor[t] = run;
    run += c;
  }
  if (tid == 0) start[T] = total;
  __syncthreads();
  for (int t = tid; t < T; t += kCsrBatchThreads) offsets[static_cast<long long>(b) * T + t] = before + start[t];
  if (b == nb - 1 && tid == 0) offsets[static_cast<long long>(nb) * T] = before + total;
  for (int s = tid; s < EK; s += kCsrBatchThreads) {
    const long long t = load_index(ind, index_dtype, static_cast<long long>(b) * EK + s);
    if (t >= 0 && t < T) list[atomicAdd(&cursor[t], 1)] = s;
  }
  __syncthreads();
  for (int s = tid; s < EK; s += kCsrBatchThreads) {
    const long long t = load_index(ind, index_dtype, static_cast<long long>(b) * EK + s);
    if (t < 0 || t >= T) continue;
    const int lo = start[t], hi = start[t + 1];
    int rank = 0;
    for (int i = lo; i < hi; ++i) rank += list[i] < s;
    entries[before + lo + rank] = b * EK + s;
  }
}

// ---- CSR by counting sort, any size ---------------------------------------------------------------------------------------
// info[0] = heaviest row, info[1] = rows touched, info[2] = 1 if an id was out of range, info[3] = valid slots
__global__ void __launch_bounds__(256) csr_count_kernel(const void* __restrict__ ind, int index_dtype, int B, int T, int E, int K,
                                                       int* __restrict__ counts, int* __restrict__ info) {
  // the four summary figures are reduced per CTA in shared memory first: one global atomic per CTA and figure
  __shared__ int s_max, s_rows, s_bad, s_valid;
  if (threadIdx.x == 0) { s_max = 0; s_rows = 0; s_bad = 0; s_valid = 0; }
  __syncthreads();
  int my_max = 0, my_rows = 0, my_valid = 0;
  const long long n = static_cast<long long>(B) * E * K;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long s = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; s < n; s += stride) {
    const long long t = load_index(ind, index_dtype, s);
    if (t < 0 || t >= T) {
      s_bad = 1;
      continue;
    }
    const long long b = s / (static_cast<long long>(E) * K);
    const int c = atomicAdd(counts + b * T + t, 1) + 1;
    my_max = max(my_max, c);
    my_rows += (c == 1);
    ++my_valid;
  }
  atomicMax(&s_max, my_max);
  atomicAdd(&s_rows, my_rows);
  atomicAdd(&s_valid, my_valid);
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicMax(info + 0, s_max);
    atomicAdd(info + 1, s_rows);
    if (s_bad) info[2] = 1;
    atomicAdd(info + 3, s_valid);
  }
}

constexpr int kScanBlock = 1024;      // rows per scan block (256 threads x 4)
// phase 1: per-block exclusive scan of counts into offsets, block totals into block_sums
__global__ void __launch_bounds__(256) csr_scan_blocks_kernel(const int* __restrict__ counts, int* __restrict__ offsets,
                                                             int* __restrict__ block_sums, long long rows) {
  __shared__ int warp_tot[8];
  const long long base = static_cast<long long>(blockIdx.x) * kScanBlock + threadIdx.x * 4;
  int v[4], sum = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[i] = (base + i < rows) ? counts[base + i] : 0;
    sum += v[i];
  }
  int incl = sum;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += o;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  int wbase = 0;
  for (int w = 0; w < warp; ++w) wbase += warp_tot[w];
  int run = wbase + incl - sum;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (base + i < rows) offsets[base + i] = run;
    run += v[i];
  }
  if (threadIdx.x == 255) block_sums[blockIdx.x] = wbase + incl;
}
// phase 2: one CTA turns block_sums into exclusive prefixes (serial over chunks of 256; the number of blocks is rows/1024)
__global__ void __launch_bounds__(256) csr_scan_sums_kernel(int* __restrict__ block_sums, int nblocks, int* __restrict__ total) {
  __shared__ int warp_tot[8];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int c0 = 0; c0 < nblocks; c0 += 256) {
    const int i = c0 + threadIdx.x;
    const int v = (i < nblocks) ? block_sums[i] : 0;
    int incl = v;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += o;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    int wbase = carry;
    for (int w = 0; w < warp; ++w) wbase += warp_tot[w];
    if (i < nblocks) block_sums[i] = wbase + incl - v;
    __syncthreads();
    if (threadIdx.x == 255) carry = wbase + incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}
// phase 3: add the block prefixes; offsets[rows] = total
__global__ void __launch_bounds__(256) csr_scan_add_kernel(int* __restrict__ offsets, const int* __restrict__ block_sums,
                                                          const int* __restrict__ total, long long rows) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < rows) offsets[i] += block_sums[i / kScanBlock];
  if (i == rows) offsets[rows] = *total;
}
// entries: every valid slot takes the next free position of its row (cursor = a zeroed copy of counts' shape)
__global__ void __launch_bounds__(256) csr_fill_kernel(const void* __restrict__ ind, int index_dtype, int B, int T, int E, int K,
                                                      const int* __restrict__ offsets, int* __restrict__ cursor,
                                                      int* __restrict__ entries) {
  const long long n = static_cast<long long>(B) * E * K;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long s = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; s < n; s += stride) {
    const long long t = load_index(ind, index_dtype, s);
    if (t < 0 || t >= T) continue;
    const long long row = (s / (static_cast<long long>(E) * K)) * T + t;
    entries[offsets[row] + atomicAdd(cursor + row, 1)] = static_cast<int>(s);
  }
}
// the positions above depend on the order the atomics ran in: sort every row's slots ascending (rows are short; one
// thread per row, insertion sort) so that the CSR - and everything computed from it - is reproducible
__global__ void __launch_bounds__(256) csr_sort_rows_kernel(const int* __restrict__ offsets, int* __restrict__ entries, long long rows) {
  const long long r = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  const int lo = offsets[r], hi = offsets[r + 1];
  for (int i = lo + 1; i < hi; ++i) {
    const int v = entries[i];
    int j = i - 1;
    while (j >= lo && entries[j] > v) {
      entries[j + 1] = entries[j];
      --j;
    }
    entries[j + 1] = v;
  }
}

template <typename TO>
__global__ void __launch_bounds__(256) compact_index_kernel(const void* __restrict__ ind, int index_dtype, long long n, long long T,
                                                           TO* __restrict__ out, int32_t* __restrict__ status) {
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long s = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; s < n; s += stride) {
    const long long t = load_index(ind, index_dtype, s);
    if ((t < 0 || t >= T) && status) atomicOr(status, EGS_STATUS_INDEX_OUT_OF_RANGE);
    out[s] = static_cast<TO>(t);
  }
}

// ---- token-major scatter from the CSR -----------------------------------------------------------------------------------
// One CTA per token row; thread j owns output columns j, j + 128, ...  For every slot of the row, in CSR order:
// acc[n] += sum_c Y[slot, c] * W(e, c, n) (+ bias[e, n]).  The Y row is staged in shared memory.
constexpr int kCsrThreads = 128;
constexpr int kCsrMaxCols = 8;        // columns per thread: N <= 1024
template <typename T>
__global__ void __launch_bounds__(kCsrThreads) csr_scatter_kernel(const T* __restrict__ Y, const T* __restrict__ W,
                                                                 const T* __restrict__ bias, const int* __restrict__ offsets,
                                                                 const int* __restrict__ entries, T* __restrict__ Out, int E,
                                                                 int K, int C, int N, int w_layout, int accumulate) {
  extern __shared__ float yrow[];       // [C]
  const long long row = blockIdx.x;
  const int lo = offsets[row], hi = offsets[row + 1];
  float acc[kCsrMaxCols];
#pragma unroll
  for (int i = 0; i < kCsrMaxCols; ++i) acc[i] = 0.f;
  for (int it = lo; it < hi; ++it) {
    const int slot = entries[it];
    const int e = (slot / K) % E;
    __syncthreads();
    for (int c = threadIdx.x; c < C; c += kCsrThreads) yrow[c] = to_f32<T>(Y[static_cast<long long>(slot) * C + c]);
    __syncthreads();
    const T* We = W + static_cast<long long>(e) * C * N;
#pragma unroll
    for (int i = 0; i < kCsrMaxCols; ++i) {
      const int n = threadIdx.x + i * kCsrThreads;
      if (n >= N) break;
      float s = bias ? to_f32<T>(bias[static_cast<long long>(e) * N + n]) : 0.f;
      if (w_layout == EGS_W_CN) {
        for (int c = 0; c < C; ++c) s = fmaf(yrow[c], to_f32<T>(We[static_cast<long long>(c) * N + n]), s);
      } else {
        const T* wr = We + static_cast<long long>(n) * C;
        for (int c = 0; c < C; ++c) s = fmaf(yrow[c], to_f32<T>(wr[c]), s);
      }
      acc[i] += s;
    }
  }
#pragma unroll
  for (int i = 0; i < kCsrMaxCols; ++i) {
    const int n = threadIdx.x + i * kCsrThreads;
    if (n >= N) break;
    const long long o = row * N + n;
    Out[o] = from_f32<T>(accumulate ? to_f32<T>(Out[o]) + acc[i] : acc[i]);
  }
}

int grid_1d(long long items, int per_block, int cap) {
  long long blocks = (items + per_block - 1) / per_block;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return static_cast<int>(blocks);
}

}  // namespace

template <int WPE, int R>
static cudaError_t launch_topk_regs(const float* scores, void* ind, int index_dtype, int B, int T, int E, int K, cudaStream_t st) {
  // experts per CTA: whole 32-byte sectors of scores, but no fewer CTAs than SMs where there are that many (batch, expert) pairs
  int eg = 16 / WPE < 8 ? 16 / WPE : 8;
  while (eg > 1 && (eg / 2 >= E || static_cast<long long>(B) * ((E + eg - 1) / eg) < 148)) eg /= 2;
  int P = 1, eg_log2 = 0;
  while (P < K) P <<= 1;
  while ((1 << eg_log2) < eg) ++eg_log2;
  const size_t turn = static_cast<size_t>(eg) * (WPE * 32 * kSelChunk + 4) * 4, lists = static_cast<size_t>(eg) * P * 8;
  const size_t smem = turn > lists ? turn : lists;
  if (smem > 48 * 1024) {      // at most 8 lists of kTopkMaxK entries
    cudaError_t err = ensure_smem_optin<route_topk_regs_kernel<WPE, R>>(8 * kTopkMaxK * 8);
    if (err != cudaSuccess) return err;
  }
  return launch_kernel(route_topk_regs_kernel<WPE, R>, B * ((E + eg - 1) / eg), eg * WPE * 32, smem, st, true, scores, ind, index_dtype, T, E, K, eg_log2, P);
}

cudaError_t launch_route_topk(const float* scores, void* ind, int index_dtype, int B, int T, int E, int K, cudaStream_t st) {
  cudaError_t err = cudaSuccess;
  if (T > 8 * 32 * kSelMaxKeys) {
    route_topk_kernel<<<B * E, kTopkThreads, 0, st>>>(scores, ind, index_dtype, B, T, E, K);
  } else {
    // Warps per expert: enough for four warps per SM in all while every thread still has eight keys, and no fewer than hold the T
    // keys.  More than that only adds barriers to the reductions: with 32 warps per SM B=32, T=2048, E=64, K=128 took 35.0 instead
    // of 27.7 us, B=64, T=1024, E=64, K=64 30.8 instead of 24.3 us; nothing measured was faster.
    int wpe = 1;
    while (wpe < 8 && (T > wpe * 32 * kSelMaxKeys || (T > wpe * 32 * 8 && static_cast<long long>(B) * E * wpe < 148 * 4))) wpe *= 2;
    int r = 8;
    while (T > wpe * 32 * r) r *= 2;
#define EGS_TOPK_R(W)                                                                          \
  do {                                                                                         \
    if (r == 8) err = launch_topk_regs<W, 8>(scores, ind, index_dtype, B, T, E, K, st);        \
    else if (r == 16) err = launch_topk_regs<W, 16>(scores, ind, index_dtype, B, T, E, K, st); \
    else if (r == 32) err = launch_topk_regs<W, 32>(scores, ind, index_dtype, B, T, E, K, st); \
    else err = launch_topk_regs<W, 64>(scores, ind, index_dtype, B, T, E, K, st);              \
  } while (0)
    if (wpe == 1) EGS_TOPK_R(1);
    else if (wpe == 2) EGS_TOPK_R(2);
    else if (wpe == 4) EGS_TOPK_R(4);
    else EGS_TOPK_R(8);
#undef EGS_TOPK_R
  }
  count_launch();
  return err != cudaSuccess ? err : cudaGetLastError();
}

size_t index_csr_scratch_ints(long long rows) { return static_cast<size_t>(rows) + static_cast<size_t>((rows + kScanBlock - 1) / kScanBlock) + 8; }

// counts [rows], offsets [rows + 1], entries [N], info [4], scratch [index_csr_scratch_ints(rows)] - all int32 on the device
cudaError_t launch_index_csr(const void* ind, int index_dtype, int B, int T, int E, int K, int* counts, int* offsets, int* entries,
                             int* info, int* scratch, cudaStream_t st) {
  const long long rows = static_cast<long long>(B) * T;
  const long long n = static_cast<long long>(B) * E * K;
  const int nblocks = static_cast<int>((rows + kScanBlock - 1) / kScanBlock);
  int* cursor = scratch;
  int* block_sums = scratch + rows;
  int* total = block_sums + nblocks;
  // one CTA per batch element where its rows and slots fit in shared memory and the partial figures in the scratch
  const long long ek = static_cast<long long>(E) * K;
  const size_t place_smem = (2 * static_cast<size_t>(T) + 1 + static_cast<size_t>(ek)) * sizeof(int);
  int4* partial = reinterpret_cast<int4*>((reinterpret_cast<uintptr_t>(scratch) + 15) & ~static_cast<uintptr_t>(15));
  if (n > 0 && rows > 0 && place_smem <= 200 * 1024 && (4ll * B + 4) * static_cast<long long>(sizeof(int)) <= static_cast<long long>(index_csr_scratch_ints(rows) * sizeof(int))) {
    cudaError_t err = ensure_smem_optin<csr_batch_place_kernel>(200 * 1024);
    if (err == cudaSuccess) err = ensure_smem_optin<csr_batch_count_kernel>(200 * 1024);
    if (err != cudaSuccess) return err;
    err = launch_kernel(csr_batch_count_kernel, B, kCsrBatchThreads, static_cast<size_t>(T) * sizeof(int), st, true, ind, index_dtype, T, static_cast<int>(ek), counts, partial);
    if (err == cudaSuccess)
      err = launch_kernel(csr_batch_place_kernel, B, kCsrBatchThreads, place_smem, st, true, ind, index_dtype, T, static_cast<int>(ek), counts, partial, offsets, entries, info);
    count_launch(2);
    return err;
  }
  cudaError_t err = launch_fill_zero(counts, static_cast<size_t>(rows) * sizeof(int), st);
  if (err == cudaSuccess) err = launch_fill_zero(info, 4 * sizeof(int), st);
  if (err == cudaSuccess) err = launch_fill_zero(cursor, static_cast<size_t>(rows) * sizeof(int), st);
  if (err != cudaSuccess) return err;
  if (n > 0) csr_count_kernel<<<grid_1d(n, 256, 148 * 8), 256, 0, st>>>(ind, index_dtype, B, T, E, K, counts, info);
  if (rows > 0) {
    csr_scan_blocks_kernel<<<nblocks, 256, 0, st>>>(counts, offsets, block_sums, rows);
    csr_scan_sums_kernel<<<1, 256, 0, st>>>(block_sums, nblocks, total);
    csr_scan_add_kernel<<<static_cast<int>((rows + 1 + 255) / 256), 256, 0, st>>>(offsets, block_sums, total, rows);
  } else {
    err = launch_fill_zero(offsets, sizeof(int), st);
    if (err != cudaSuccess) return err;
  }
  if (n > 0) {
    csr_fill_kernel<<<grid_1d(n, 256, 148 * 8), 256, 0, st>>>(ind, index_dtype, B, T, E, K, offsets, cursor, entries);
    csr_sort_rows_kernel<<<static_cast<int>((rows + 255) / 256), 256, 0, st>>>(offsets, entries, rows);
  }
  count_launch(n > 0 ? 6 : 3);
  return cudaGetLastError();
}

cudaError_t launch_compact_index(const void* ind, int index_dtype, long long n, long long T, void* out, int out_dtype,
                                 int32_t* status, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const int grid = grid_1d(n, 256, 148 * 8);
  if (out_dtype == EGS_I64) compact_index_kernel<long long><<<grid, 256, 0, st>>>(ind, index_dtype, n, T, static_cast<long long*>(out), status);
  else if (out_dtype == EGS_I32) compact_index_kernel<int><<<grid, 256, 0, st>>>(ind, index_dtype, n, T, static_cast<int*>(out), status);
  else compact_index_kernel<short><<<grid, 256, 0, st>>>(ind, index_dtype, n, T, static_cast<short*>(out), status);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_csr_scatter(const void* Y, const void* W, const void* bias, const int* offsets, const int* entries, void* Out,
                               long long rows, int E, int K, int C, int N, int w_layout, int accumulate, int dtype,
                               cudaStream_t st) {
  if (rows == 0 || N == 0) return cudaSuccess;
  const size_t smem = static_cast<size_t>(C) * sizeof(float);
  const unsigned grid = static_cast<unsigned>(rows);
#define EGS_CSR(TY)                                                                                                       \
  csr_scatter_kernel<TY><<<grid, kCsrThreads, smem, st>>>(static_cast<const TY*>(Y), static_cast<const TY*>(W),           \
                                                        static_cast<const TY*>(bias), offsets, entries, static_cast<TY*>(Out), \
                                                        E, K, C, N, w_layout, accumulate)
  if (dtype == EGS_F32) EGS_CSR(float);
  else if (dtype == EGS_F16) EGS_CSR(__half);
  else EGS_CSR(__nv_bfloat16);
#undef EGS_CSR
  count_launch();
  return cudaGetLastError();
}

}  // namespace egs

// Internal declarations shared by the kernel files and the C-ABI file of libegs_b200.so.
//
// Vocabulary used across the kernels:
//   slot        one routed token slot (b, e, k); its linear id is (b*E + e)*K + k
//   token row   row b*T + t of a [B,T,F] tensor (X, Out, dX, dOut), t = Ind[slot]
//   slot row    row `slot` of a [B,E,K,F] tensor (Y, dY)
//   expert row  m in [0, B*K): the m-th slot of one expert, b = m / K, k = m % K
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/egs_b200.h"

namespace egs {

// ------------------------------------------------------------------------------------------------
// element conversion
// ------------------------------------------------------------------------------------------------
template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Reads Ind[pos] for any of the three index widths.
__device__ __forceinline__ long long load_index(const void* ind, int index_dtype, long long pos) {
  if (index_dtype == EGS_I64) return static_cast<const long long*>(ind)[pos];
  if (index_dtype == EGS_I32) return static_cast<const int*>(ind)[pos];
  return static_cast<const short*>(ind)[pos];
}

// The caller's status word and, where one was registered for it (egs_set_status_mirror), its mapped host mirror.  A CTA that
// gives up (a wait that ran out, misaligned shared memory) stores the reason there on its way out - rare, and the host looks
// before its next call, so that no copy of the word has to be queued behind every pass.
struct StatusRef {
  int32_t* word = nullptr;
  int32_t* mirror = nullptr;
  __device__ __forceinline__ bool timed_out() const {
    return word && (*reinterpret_cast<volatile int32_t*>(word) & EGS_STATUS_PIPELINE_TIMEOUT);
  }
  __device__ __forceinline__ void report(int bits) const {
    if (word) atomicOr(word, bits);
  }
  __device__ __forceinline__ void tell_host() const {
    if (word && mirror)
      *reinterpret_cast<volatile int32_t*>(mirror) =
          *reinterpret_cast<volatile int32_t*>(word) & (EGS_STATUS_PIPELINE_TIMEOUT | EGS_STATUS_INTERNAL);
  }
};
StatusRef status_ref(int32_t* status_word);

// Division of 0 <= n < 2^31 by a divisor known on the host: a multiplication, an addition and a shift (Granlund and Montgomery, "Division by
// invariant integers using multiplication").  The compiler's sequence for a divisor it does not know takes 100 clocks and more, and ten
// of those stood one after the other at the start of every role of the persistent kernels.
struct Div {
  uint32_t mul = 1, shift = 0;
  int d = 1;
  Div() = default;
  explicit Div(int divisor) : d(divisor) {
    while ((1ll << shift) < divisor) ++shift;
    mul = static_cast<uint32_t>((((1ull << shift) - static_cast<uint64_t>(divisor)) << 32) / static_cast<uint64_t>(divisor)) + 1u;
  }
  __device__ __forceinline__ int quotient(int n) const { return static_cast<int>((__umulhi(mul, static_cast<uint32_t>(n)) + static_cast<uint32_t>(n)) >> shift); }
  // divides n, returns the remainder
  __device__ __forceinline__ int remainder(int& n) const {
    const int q = quotient(n), r = n - q * d;
    n = q;
    return r;
  }
};

// ------------------------------------------------------------------------------------------------
// parameter blocks (validated on the host: every product below fits in int32 unless typed int64)
// ------------------------------------------------------------------------------------------------

// The plan of a scatter with 16-bit tensors on the tensor cores, words on the device: whether its token rows accumulate in the float32 rows
// (else additions go straight into the 16-bit output); for each column tile the units that have been added (zero at first).
enum PlanWords { kPlanHot = 0, kPlanAdded = 1, kPlanWords = 64 };

struct RowGemmParams {
  const void* A;      // G: token rows [B*T, C]      S: slot rows [B*E*K, C]
  const void* W;      // [E, C, N] (EGS_W_CN) or [E, N, C] (EGS_W_NC)
  const void* Ind;    // [B, E, K]
  void* Out;          // G: slot rows [B*E*K, N]     S: token rows [B*T, N]
  float* acc;         // S with 16-bit tensors: float32 accumulation rows [B*T, N]; otherwise unused
  int* plan;          // 16-bit S on the tensor cores: PlanWords
  int rounds;         // ... and whether the kernel rounds the float32 rows itself
  const void* bias;   // optional [E, N] in the tensors' dtype: bias[e, :] is added to every produced row of expert e
                      // (G: to the stored row; S: to the row before it is added to its token row); NULL = none
  StatusRef status;    // optional device status word
  int B, T, E, K, C, N;
  int M;              // expert rows per expert = B*K
  int w_layout;
  int index_dtype;
  int BN;             // tensor path: tile width over N (multiple of 16, <= 256)
  int stages;         // tensor path: pipeline depth
  int expert_fastest; // tensor path: grid order (1: experts vary fastest, row tiles slowest)
  int row_tiles;      // tensor path: 128-row accumulator tiles per CTA (1 or 2)
  int persistent;     // tensor path: 1 = persistent warp-specialised variant
  int pair;           // 16-bit G, S: tiles of 256 rows on pairs of SMs
  int tile_group;     // 16-bit S: column tiles that a row block stays in shared memory for (0: it is loaded for each)
  int full_waves;     // ... and waves of row blocks that stay for all of them
  int slot_boxes;     // 16-bit and strict float32 S: slot rows come as TMA boxes
  int after_own;      // launched behind a kernel of the same call (fill, preparation): see launch_kernel
};

struct DWeightParams {
  const void* Xsrc;   // token rows [B*T, FG]  (gathered through Ind)
  const void* Ysrc;   // slot rows  [B*E*K, FD]
  const void* Ind;
  void* out;          // final output in the tensors' dtype
  float* acc;         // fp32 accumulation buffer when splits > 1 (may alias out for fp32), else unused
  StatusRef status;
  int B, T, E, K, FG, FD;
  int M;              // B*K
  int out_layout;
  int index_dtype;
  int splits;         // number of row ranges the contraction is split into
  int rows_per_split; // multiple of the stage depth
  int BN;             // tensor path: tile width over FD
  int stages;
  int row_tiles;      // tensor path: 128-feature accumulator tiles per CTA over FG (1 or 2)
  int after_own;      // launched behind the fill of `acc`: see launch_kernel
  int swap;           // 16-bit: the slot rows' features run along the accumulator's rows
  int pair;           // 16-bit: tiles of 256 rows on pairs of SMs
  int slot_boxes;     // 16-bit and strict float32: slot rows come as TMA boxes
};

// Fused pair G -> S (tensor path only):  Mid = gather(Src) x W1[e] is stored as slot rows AND fed, without leaving the
// SM (shared memory for float32 tensors, tensor memory for 16-bit ones), into  Dst[token rows] += Mid x W2[e].
struct FusedParams {
  const void* Src;     // token rows [B*T, C1]
  const void* W1;      // [E, C1, N1] (EGS_W_CN) or [E, N1, C1] (EGS_W_NC)
  const void* W2;      // [E, N1, N2] (EGS_W_CN) or [E, N2, N1] (EGS_W_NC)
  const void* Ind;     // [B, E, K]
  void* Mid;           // slot rows [B*E*K, N1], overwritten
  float* Dst;          // float32 token rows [B*T, N2], added to (16-bit tensors: the accumulation rows of the scratch)
  void* Out16;         // 16-bit tensors: the output token rows [B*T, N2] that direct 16-bit additions go to
  const int* plan;     // 16-bit tensors: device flag, non-zero = token rows accumulate in the float32 rows, zero = direct additions
  StatusRef status;
  int B, T, E, K, C1, N1, N2;
  int M;               // B*K
  int w_layout;        // of both weights
  int index_dtype;
  int BN1, BN2;        // MMA widths (multiples of 16)
  int stages;
  int expert_fastest;  // 16-bit kernel: order of the row blocks a CTA walks (1: experts vary fastest)
  int after_own;       // launched behind a kernel of the same call (fill, preparation): see launch_kernel
  uint32_t slot_bytes; // 16-bit kernel: bytes of one ring slot
};

// ------------------------------------------------------------------------------------------------
// launchers implemented in the kernel files; each returns a cudaError_t from the launch
// ------------------------------------------------------------------------------------------------
cudaError_t launch_generic_rowgemm(const RowGemmParams& p, bool scatter, int dtype, cudaStream_t st);
void configure_generic_dweight(DWeightParams& p);   // tile (BN, row_tiles in units of 32 features) and row ranges
cudaError_t launch_generic_dweight(const DWeightParams& p, int dtype, cudaStream_t st);
// out[e, n] = sum over the slots of expert e of a row of Src: token rows through Ind, or slot rows where Ind is NULL
cudaError_t launch_expert_row_sum(const void* Src, const void* Ind, int index_dtype, void* out, int B, int T, int E, int K, int N,
                                  int dtype, StatusRef status, cudaStream_t st);
// early: dependents may start with this kernel; false in front of and behind the generic kernels (see the top of egs_generic.cu)
cudaError_t launch_fill_zero(void* ptr, size_t bytes, cudaStream_t st, bool early = true);
cudaError_t launch_convert_from_f32(const float* src, void* dst, size_t n, int dtype, cudaStream_t st, bool early);
cudaError_t launch_convert_to_f32(const void* src, float* dst, size_t n, int dtype, cudaStream_t st);
// 16-bit scatter (see egs_generic.cu): prepare decides between direct additions (no token row gets more than `limit` contributions)
// and float32 rows, and zeroes (or seeds) what the additions go to; finish rounds the float32 rows for kernels that do not do that.
// csr_info: the summary of a prepared CSR, whose heaviest row decides; NULL = the ids are counted.  flags: scratch of B ints.
cudaError_t launch_scatter_prepare(const void* Ind, int index_dtype, int B, int T, int E, int K, const int* csr_info, int limit, int* flags,
                                   int* plan, float* acc, void* out16, int N, int zero_output, int dtype, StatusRef status, cudaStream_t st);
cudaError_t launch_scatter_finish(const int* plan, const float* acc, void* out16, size_t n, int dtype, cudaStream_t st);

// Tensor-core (tcgen05) family.  `configure_*` fills BN/stages and returns the dynamic shared memory size.
size_t configure_tensor_rowgemm(RowGemmParams& p, bool scatter);
size_t configure_tensor_dweight(DWeightParams& p);
cudaError_t launch_tensor_rowgemm(const RowGemmParams& p, bool scatter, size_t smem_bytes, cudaStream_t st);
cudaError_t launch_tensor_dweight(const DWeightParams& p, size_t smem_bytes, cudaStream_t st);

// 16-bit tensors (egs_dense16.cu): persistent kernels for G, S and D.
void configure_dense16_rowgemm(RowGemmParams& p, bool scatter);
// G as configured: units of half a tile in the last wave, columns of the first half (see plan_tail)
void dense16_half_tiles(const RowGemmParams& p, int* units, int* first);
cudaError_t launch_dense16_rowgemm(const RowGemmParams& p, bool scatter, int dtype, cudaStream_t st);
void configure_dense16_dweight(DWeightParams& p);
cudaError_t launch_dense16_dweight(const DWeightParams& p, int dtype, cudaStream_t st);

// Strict float32 (egs_strict.cu).  Long contractions are fine up to kStrictMaxContraction (see run_rowgemm).
void configure_strict_rowgemm(RowGemmParams& p, bool scatter);
cudaError_t launch_strict_rowgemm(const RowGemmParams& p, bool scatter, cudaStream_t st);
void configure_strict_dweight(DWeightParams& p);
cudaError_t launch_strict_dweight(const DWeightParams& p, cudaStream_t st);

// Fused pair: `configure` returns 0 when the shape does not fit the kernel (the caller then runs G and S).
size_t configure_tensor_fused_pair(FusedParams& p, int precision);
cudaError_t launch_tensor_fused_pair(const FusedParams& p, int precision, size_t smem_bytes, cudaStream_t st);
// Operator G on pairs of SMs (egs_gather2.cu, EGS_PATH_PAIRED): fills BN / stages, returns the shared memory size or 0.
size_t configure_tensor_gather2(RowGemmParams& p);
cudaError_t launch_tensor_gather2(const RowGemmParams& p, int dtype, size_t smem_bytes, cudaStream_t st);
// Fused pair for 16-bit tensors (persistent kernel, egs_pair16.cu); same conventions as the float32 one.
size_t configure_tensor_pair16(FusedParams& p);
cudaError_t launch_tensor_pair16(const FusedParams& p, int dtype, size_t smem_bytes, cudaStream_t st);

// Opaque 128-byte TMA tensor map (CUtensorMap of the driver API) and its encoder for a dense tensor of 16-bit elements of up to
// four dimensions, dims[0] innermost, 128-byte swizzle, out-of-range elements read as zero.  Returns false when the driver
// refuses the geometry (strides must be multiples of 16 bytes, box sides at most 256).
struct alignas(64) TensorMap3 {
  unsigned char bytes[128];
};
bool encode_tensor_map_16bit(TensorMap3* out, const void* base, int rank, const unsigned long long* dims, const unsigned* box);
// ... of up to five dimensions whose strides (bytes, of all but the first) are given
bool encode_tensor_map_16bit_strided(TensorMap3* out, const void* base, int rank, const unsigned long long* dims, const unsigned long long* strides,
                                     const unsigned* box);
// The same for 32-bit elements.  kMapSwizzle128Base32: the XOR of the 128-byte swizzle acts on 32-byte pairs of chunks with the row modulo 4.
enum { kMapSwizzleNone = 0, kMapSwizzle128 = 1, kMapSwizzle128Base32 = 2 };
bool encode_tensor_map_32bit(TensorMap3* out, const void* base, int rank, const unsigned long long* dims, const unsigned* box, int swizzle);

// Index preparation (egs_index.cu).  All index arrays are int32 on the device.
cudaError_t launch_route_topk(const float* scores, void* ind, int index_dtype, int B, int T, int E, int K, cudaStream_t st);
size_t index_csr_scratch_ints(long long rows);
cudaError_t launch_index_csr(const void* ind, int index_dtype, int B, int T, int E, int K, int* counts, int* offsets, int* entries,
                             int* info, int* scratch, cudaStream_t st);
cudaError_t launch_compact_index(const void* ind, int index_dtype, long long n, long long T, void* out, int out_dtype,
                                 int32_t* status, cudaStream_t st);
cudaError_t launch_csr_scatter(const void* Y, const void* W, const void* bias, const int* offsets, const int* entries, void* Out,
                               long long rows, int E, int K, int C, int N, int w_layout, int accumulate, int dtype,
                               cudaStream_t st);

// Bounded-wait self-test (see the kernel): out = two ints on the device.
cudaError_t launch_wait_timeout_selftest(int32_t* status, int* out, long long limit_cycles, cudaStream_t st);

void count_launch(int n = 1);

// ------------------------------------------------------------------------------------------------
// Programmatic dependent launch.  A kernel launched with `dependent` may become resident as soon as every CTA of the kernel before it
// on the stream has called pdl_trigger or exited; pdl_wait returns when that kernel has finished and its writes are visible.  A
// kernel behind anything else, or launched without the attribute, returns from pdl_wait at once.  The rules that keep this sound:
//   * a kernel launched with the attribute calls pdl_wait in every launch, on its way out of an abort too: that it has finished then
//     means that everything before it has;
//   * it calls pdl_wait before it touches global memory, except where the kernel before it belongs to the same call (after_own: a
//     fill, the scatter's preparation): that one calls pdl_wait BEFORE pdl_trigger, so that all that came before it is visible to
//     its dependent from the start, which then only waits before it touches what the fill or the preparation wrote.  A preparation
//     behind its call's counting kernel, which has waited before it triggered, may trigger at once: the scatter's contraction then
//     runs under the counting too (4 batch elements of 16380 ids: 115 us a pass if not, 106 so).
//   * it takes no `__restrict__` pointers: until the wait its inputs may still be written, and loads that are promised the contrary are
//     not bound by it.  (Row sums, which are launched normally, keep theirs.  Without them nothing got slower by more than the runs differ.)
// Launch and set-up of a kernel so run under the end of the one before, also across calls: 1-2 us a kernel (a training pass of ten
// kernels 151 -> 145 us, one of fourteen 253 -> 249).  The persistent kernels trigger when their last tile has been issued: triggering
// at their start lets a dependent's waiting CTAs keep a kernel of another stream off an SM.  Kernels of which an SM holds several CTAs
// (egs_generic.cu) do not trigger at all.  Ordinary launches: the bias row sums, the TF32 and fused kernels that no fill of their call precedes,
// egs_gather2.cu, top-k of long sequences, the CSR of large batches and what reads it.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... Params, class... Args>
cudaError_t launch_kernel(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, bool dependent, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// The opt-in to large dynamic shared memory is per kernel function and device: done once per thread and device, for `bytes`.
template <auto kernel>
cudaError_t ensure_smem_optin(int bytes) {
  static thread_local int done_device = -1;
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  if (done_device == dev) return cudaSuccess;
  err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (err == cudaSuccess) done_device = dev;
  return err;
}

}  // namespace egs

// Host runtime shared by the C-ABI entry points: per-device context, tensor-map cache, GEMM launcher.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/toner_b200.h"
#include "gemm_tcgen05.cuh"

namespace toner {

// Return codes of the C-ABI (0 = ok, > 0 = host-side argument / runtime error).
enum : int {
  kErrArg = 1,         // null / misaligned pointer, bad size
  kErrCuda = 2,        // a CUDA runtime call failed (see toner_last_error)
  kErrDriver = 3,      // cuTensorMapEncodeTiled unavailable or failed
  kErrWorkspace = 4,   // caller-provided workspace too small
  kErrUnsupported = 5  // shape or option outside what the kernels cover
};

void set_error(const std::string& msg);
int fail(int code, const std::string& msg);

#define TONER_CUDA(expr)                                                                         \
  do {                                                                                           \
    cudaError_t err__ = (expr);                                                                  \
    if (err__ != cudaSuccess)                                                                    \
      return ::toner::fail(::toner::kErrCuda, std::string(#expr) + ": " + cudaGetErrorString(err__)); \
  } while (0)

struct Context {
  int device = -1;
  int num_sms = 0;
  int gemm_sms = 0;  // CTAs the persistent GEMM may occupy (toner_set_gemm_sm_limit)
  int gemm_wide_kb = 80;  // k-blocks (all plane products together) from which 256 x 512 tiles are considered
  CUtensorMap* arena_dev = nullptr;   // tensor maps live here; slots are never rewritten between resets
  CUtensorMap* arena_host = nullptr;  // pinned mirror used as the copy source
  int arena_cap = 0, arena_used = 0;
  int* status_dev = nullptr;          // set by a kernel whose bounded wait ran out
  unsigned long long* prof_dev = nullptr;  // eight cycle counters, allocated when phase profiling is switched on
  void* map_cache = nullptr;          // operand description -> arena slot and upload event (runtime.cu)
};

// Number of kernels this library has launched (all devices, all streams).
void count_launch(int n = 1);

// Launch with programmatic stream serialisation: the kernel's blocks may be scheduled while the previous kernel of the
// stream drains; each kernel orders itself with ptx::pdl_begin().  Launch latency and prologue (barriers, tensor memory,
// descriptors) of a chain of short products then hide behind one another.  `cluster`: blocks per cluster (0: none).
template <typename... P, typename... A>
cudaError_t launch(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream, int cluster, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster > 0 ? cluster : 1;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 0 ? 2 : 1;
  count_launch();
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
#define TONER_LAUNCH(kernel, grid, threads, stream, ...) TONER_CUDA(launch(kernel, dim3(grid), threads, 0, stream, 0, __VA_ARGS__))

// Shared-memory limits of the factor engine's kernels on the current device; false where they were refused.
bool allow_factor_kernels();

// Context of the current device (created on first use).  Returns nullptr and sets the error on failure.
Context* context();

// Device pointer to `batch` consecutive tensor maps describing the separately allocated matrices of op.list (an operand
// that is one stack needs no map in memory: its map travels with the launch).  box_rows is the outer box extent for K-major operands (tile rows); MN-major
// operands always use 64 x 64 boxes.
int get_maps(Context* ctx, const toner_operand& op, int batch, int box_rows, cudaStream_t stream, const CUtensorMap** out);

// skip: optional, per batch (device memory): the product is left out where it is not zero.  half_in, half_out: both operands, and
// the operand planes of the result, are symmetric matrices of which only the 256 x 256 blocks on and above the diagonal are stored.
struct GemmMore {
  const int* skip = nullptr;
  bool half_in = false, half_out = false;
};
int launch_gemm(const toner_gemm_desc& d, cudaStream_t stream, const GemmMore& more = GemmMore());
// The products of a whole polar iteration (Gram of either operand copy, polynomial, update either way and the last one) in one
// launch; claim and done[batch] are zero when it starts.  in_step: the host has launches of its own to make meanwhile.
// *taken = false: not done, the products are to be launched one by one.
int launch_polar_chain(const toner_gemm_desc (&ops)[6], int steps, bool in_step, unsigned int* claim, unsigned int* done,
                       cudaStream_t stream, bool* taken);
// Scratch (split_ws) with which launch_gemm would divide the accumulation of this product among several units; 0: none.
size_t gemm_split_bytes(const toner_gemm_desc& d);

// FP16 hi/lo split of an FP32 stack (see toner_split16).  inv_mul: per-matrix factors of the inverse scales; hi_only: the lo
// planes are not written; scratch_zeroed: the maximum accumulators in `scratch` are zero already.
int split16(const float* x, const float* const* x_list, int batch, int rows, int cols, long long ld, long long bs,
            float aff_a, float aff_b, const uint32_t* maxabs, void* scratch, void* planes, float* inv_scale,
            cudaStream_t stream, const float* inv_mul = nullptr, bool hi_only = false, bool scratch_zeroed = false);

// out[b] = sum of squares of matrix b, bitwise reproducible.  scratch: sumsq_scratch_bytes(batch).
size_t sumsq_scratch_bytes(int batch);
// (out == nullptr: only the kSumsqBlocks partial sums of each matrix are left in scratch)
constexpr int kSumsqBlocks = 296;  // two per SM on a 148-SM part; fixed so that results do not depend on the device
int sumsq_det(const float* x, int batch, int rows, int cols, long long ld, long long bs, float* scratch, float* out,
              cudaStream_t stream);

// Sum of a matrix's partial sums, added one after the other in their order; called by one warp, every lane gets the total.
// (The lanes fetch them together: the additions then run at register speed, not one load apart.)
__device__ __forceinline__ float sumsq_total(const float* __restrict__ partial, int lane) {
  constexpr int kRows = (kSumsqBlocks + 31) / 32;
  float p[kRows];
#pragma unroll
  for (int i = 0; i < kRows; ++i) p[i] = (i * 32 + lane < kSumsqBlocks) ? partial[i * 32 + lane] : 0.f;
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
#pragma unroll 8
    for (int l = 0; l < 32; ++l) t += __shfl_sync(0xffffffffu, p[i], l);
  }
  return t;
}

// Block-wide max of non-negative values into one FP32-bits accumulator: one atomic per block, and none when the
// accumulator already holds as much (thousands of blocks share a few addresses; per-warp atomics serialise in L2).
// Every thread of a 256-thread block calls this.
__device__ __forceinline__ void block_atomic_max(float v, unsigned int* acc) {
  __shared__ float warp_max[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float m = warp_max[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) m = fmaxf(m, warp_max[w]);
    const unsigned int bits = __float_as_uint(m);
    if (bits > *reinterpret_cast<volatile unsigned int*>(acc)) atomicMax(acc, bits);
  }
}

// k-blocks per accumulation chain used for FP32-accurate (split-precision) products
constexpr int kPromoteAccurate = 2;
// chain length where a relative error of 1e-6 only propagates linearly (products applied to X, W, gradients)
constexpr int kPromoteLinear = 8;

}  // namespace toner

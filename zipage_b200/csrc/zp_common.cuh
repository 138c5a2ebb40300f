// Shared device/host helpers of libzipage_b200 (sm_100a only).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/zipage_b200.h"

namespace zp {

// ---- error reporting (no exceptions cross the C boundary) -----------------
void set_error(const char* fmt, ...);
int check_launch(const char* what);

#define ZP_REQUIRE(cond, ...)            \
  do {                                   \
    if (!(cond)) {                       \
      zp::set_error(__VA_ARGS__);        \
      return ZP_ERR_INVALID_ARGUMENT;    \
    }                                    \
  } while (0)

// ---- element types ---------------------------------------------------------
template <typename T> struct Elem;
template <> struct Elem<__nv_bfloat16> {
  static __device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 from_f32(float v) { return __float2bfloat16_rn(v); }
};
template <> struct Elem<__half> {
  static __device__ __forceinline__ float to_f32(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half from_f32(float v) { return __float2half_rn(v); }
};
template <> struct Elem<float> {
  static __device__ __forceinline__ float to_f32(float v) { return v; }
  static __device__ __forceinline__ float from_f32(float v) { return v; }
};

// Round an fp32 value to T and bring it back: the value a tensor of dtype T would hold.
template <typename T> __device__ __forceinline__ float round_to(float v) {
  return Elem<T>::to_f32(Elem<T>::from_f32(v));
}

static inline size_t dtype_size(int dtype) {
  return dtype == ZP_DTYPE_F32 ? 4 : 2;
}

// Dispatch a templated launcher on the dtype code.
#define ZP_DISPATCH_DTYPE(dtype, T, ...)                                  \
  do {                                                                    \
    if ((dtype) == ZP_DTYPE_BF16) { using T = __nv_bfloat16; __VA_ARGS__; } \
    else if ((dtype) == ZP_DTYPE_F16) { using T = __half; __VA_ARGS__; }  \
    else if ((dtype) == ZP_DTYPE_F32) { using T = float; __VA_ARGS__; }   \
    else { zp::set_error("unknown dtype code %d", (int)(dtype)); return ZP_ERR_INVALID_ARGUMENT; } \
  } while (0)

// ---- block-table encoding ---------------------------------------------------
// -1 = padding, id >= 0 = ordinary page, -(id)-2 = the sequence's last page.
struct PageRef {
  int id;      // decoded page id (undefined when !valid)
  bool valid;
  bool last;
};
__device__ __forceinline__ PageRef decode_page(int entry) {
  PageRef r;
  r.valid = entry != -1;
  r.last = entry < -1;
  r.id = r.last ? (-entry - 2) : entry;
  return r;
}

// ---- reductions ---------------------------------------------------------------
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ int warp_sum_i(int v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide reductions with a fixed combination order (deterministic).  `red` is
// shared scratch of at least 32 floats; all threads of the block must call.
__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float r = (lane < nw) ? red[lane] : -INFINITY;
  r = warp_max(r);
  return r;
}
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float r = (lane < nw) ? red[lane] : 0.f;
  r = warp_sum(r);
  return r;
}

// ---- blocks of a thread-block cluster ----------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t cluster_size() { uint32_t r; asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// a float of the same shared-memory variable in another block of the cluster
__device__ __forceinline__ float ld_cluster(const float* p, uint32_t rank) {
  uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p)), ra;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(ra) : "memory");
  return v;
}

// and the way back
__device__ __forceinline__ void st_cluster(float* p, uint32_t rank, float v) {
  uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p)), ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(ra), "f"(v) : "memory");
}

// ---- kernels that begin while the one before them ends ----------------------------------------------
// A kernel launched by `launch_early` may start as soon as every block of the kernel before it on the stream has called
// `let_next_begin` or is done.  All of its threads call `wait_for_previous` first: before it, nothing may be read that an
// earlier kernel writes, and nothing written; and what earlier kernels wrote is not read through the read-only path (no
// __restrict__ const pointers).  `let_next_begin` comes after the wait, so at most two kernels of a stream overlap, and
// a kernel launched the ordinary way still waits for everything before it.  It hides the launch and the first latencies of a
// step's small kernels: a step of 4 sequences and 4 layers as a graph 197 -> 176 us, a step's attention for 192 sequences 285 -> 282.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_begin() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename... P, typename... A>
static inline cudaError_t launch_early(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// ---- 16-byte vector copies ------------------------------------------------------------------
__device__ __forceinline__ int4 ld16(const void* p) { return *reinterpret_cast<const int4*>(p); }
__device__ __forceinline__ void st16(void* p, int4 v) { *reinterpret_cast<int4*>(p) = v; }

}  // namespace zp

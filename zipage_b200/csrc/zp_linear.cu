// out = x weight^T (+ bias) for the few rows of a decode step: 16-bit tensors, fp32 accumulation, one rounding.
//
// Bound by latency: the weights of a small model are a few MB, which a library product of a few rows reads in 5 to 8 us.  Here a block has
// 16 rows of the weight and its eight warps split the inner dimension, so that even a small weight is spread over many
// SMs with all its loads in flight; and the weight is requested from HBM while the kernel before this one ends.  Products
// on mma.sync m16n8k16 (the weight's rows are the 16-row operand, eight rows of x the other).  The order of the inner dimension is
// free as long as both operands agree: a lane's 16-byte load of eight consecutive elements is its part of two k-steps, and no shared
// memory is needed before the sums of the warps meet.
//
// All of a warp's loads are issued before its first product: a second round is another trip to L2, which no other block of the SM
// covers.  Left to itself the compiler moves loads behind the first products, which wait for their own, and saves the registers.
// 8 rows, bf16, weights not in L2, launches back to back (us, cuBLAS): 2048 x 1024 2.2 (5.1), 4096 x 1024 3.2 (5.5), 6144 x 1024 3.6 (5.3), 1024 x 2048
// 2.6 (6.8), 1024 x 3072 3.8 (8.8), 2048 x 4096 5.2 (11.0).  With the loads left to the compiler, four steps at a time: 3.1, 3.6, 4.5, 4.5, 6.3 and 9.5;
// with 16 warps instead the last three 3.2, 4.5 and 6.0, and other roundings.  Without the request ahead 2048 x 1024 took 1 us more.
#include "zp_mma.cuh"

namespace zp {

constexpr int LIN_WARPS = 8;

// DEEP: 32-element steps whose loads are in flight together
template <typename T, int DEEP>
__global__ void __launch_bounds__(LIN_WARPS * 32)
small_linear_kernel(const T* x, int64_t x_stride, const T* weight, const T* bias, T* out,
                    int rows, int n_out, int k) {
  __shared__ float part[LIN_WARPS][16][9];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
  const int n0 = blockIdx.x * 16;
  // the block's rows of the weight on their way to L2 while the kernel before this one ends
  if (threadIdx.x == 0)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(weight + (int64_t)n0 * k), "r"(min(16, n_out - n0) * k * 2) : "memory");
  wait_for_previous();
  let_next_begin();
  // (rows past the end repeat the last one and are not stored)
  const T* w0 = weight + (int64_t)min(n0 + g, n_out - 1) * k + tq * 8;
  const T* w1 = weight + (int64_t)min(n0 + g + 8, n_out - 1) * k + tq * 8;
  const T* xr = x + (int64_t)min(g, rows - 1) * x_stride + tq * 8;
  const int steps = k / 32, s_end = (warp + 1) * steps / LIN_WARPS;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int s = warp * steps / LIN_WARPS; s < s_end; s += DEEP) {
    int4 a0[DEEP], a1[DEEP], b[DEEP];
#pragma unroll
    for (int d = 0; d < DEEP; ++d) {
      const int at = min(s + d, s_end - 1) * 32;
      a0[d] = ld16(w0 + at);
      a1[d] = ld16(w1 + at);
      b[d] = ld16(xr + at);
    }
    __syncwarp();      // (no load moves behind this)
#pragma unroll
    for (int d = 0; d < DEEP; ++d) {
      if (s + d >= s_end) break;
      const uint32_t lo[4] = {(uint32_t)a0[d].x, (uint32_t)a1[d].x, (uint32_t)a0[d].y, (uint32_t)a1[d].y};
      const uint32_t hi[4] = {(uint32_t)a0[d].z, (uint32_t)a1[d].z, (uint32_t)a0[d].w, (uint32_t)a1[d].w};
      mma16816<T>(acc, lo, (uint32_t)b[d].x, (uint32_t)b[d].y);
      mma16816<T>(acc, hi, (uint32_t)b[d].z, (uint32_t)b[d].w);
    }
  }
  part[warp][g][2 * tq] = acc[0];
  part[warp][g][2 * tq + 1] = acc[1];
  part[warp][g + 8][2 * tq] = acc[2];
  part[warp][g + 8][2 * tq + 1] = acc[3];
  __syncthreads();
  const int n = threadIdx.x & 15, r = threadIdx.x >> 4;
  if (r < rows && n0 + n < n_out) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < LIN_WARPS; ++w) v += part[w][n][r];
    if (bias) v += Elem<T>::to_f32(bias[n0 + n]);
    out[(int64_t)r * n_out + n0 + n] = Elem<T>::from_f32(v);
  }
}

}  // namespace zp

extern "C" int zp_small_linear(const void* x, int64_t x_stride, const void* weight, const void* bias, void* out, int rows, int n_out, int k,
                               int dtype, void* stream) {
  if (rows == 0 || n_out == 0) return ZP_OK;
  ZP_REQUIRE(x && weight && out, "zp_small_linear: null pointer");
  // (sizes up to which the bytes of a block's rows and the number of blocks are counted in 32 bits)
  ZP_REQUIRE(rows > 0 && rows <= 8 && n_out > 0 && n_out <= 1 << 30 && k > 0 && k <= 1 << 24 && k % 32 == 0 && x_stride % 8 == 0,
             "zp_small_linear: sizes not supported");
  ZP_REQUIRE(((uintptr_t)x | (uintptr_t)weight) % 16 == 0, "zp_small_linear: x and weight must be 16-byte aligned");
  auto run = [&](auto t) {
    using T = decltype(t);
    const int blocks = (n_out + 15) / 16;
    auto go = [&](auto kernel) {
      zp::launch_early(kernel, dim3(blocks), zp::LIN_WARPS * 32, 0, (cudaStream_t)stream, (const T*)x, x_stride, (const T*)weight, (const T*)bias, (T*)out,
                       rows, n_out, k);
    };
    // A warp's steps at once, as registers allow: all of them while a block has an SM to itself (up to 222 registers a thread; 1024 x 3072 3.5 us for
    // 3.9 with half of them, 4 rows), half of them where two have to share it (2720 x 3072 5.2 for 6.3).  No more than there are: the others would be loads
    // of the last one again (32768 x 256 5.6 us for 9.2 with four).
    const bool alone = blocks <= 148;
    if (k <= 256) go(zp::small_linear_kernel<T, 1>);
    else if (k <= 512) go(zp::small_linear_kernel<T, 2>);
    else if (k <= 768) go(zp::small_linear_kernel<T, 3>);
    else if (k <= 1024) go(zp::small_linear_kernel<T, 4>);
    else if (k <= 1536) go(zp::small_linear_kernel<T, 6>);
    else if (k <= 2048) go(zp::small_linear_kernel<T, 8>);
    else if (k <= 3072) alone ? go(zp::small_linear_kernel<T, 12>) : go(zp::small_linear_kernel<T, 6>);
    else alone ? go(zp::small_linear_kernel<T, 16>) : go(zp::small_linear_kernel<T, 8>);
  };
  if (dtype == ZP_DTYPE_BF16) run(__nv_bfloat16());
  else if (dtype == ZP_DTYPE_F16) run(__half());
  else { zp::set_error("zp_small_linear: 16-bit tensors only"); return ZP_ERR_UNSUPPORTED; }
  return zp::check_launch("zp_small_linear");
}

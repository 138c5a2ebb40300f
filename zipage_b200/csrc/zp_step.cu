// The small per-step ops around the attention path of one decoder layer, and the decode
// bookkeeping, as single launches:
//   * RMSNorm with optional residual add,
//   * SiLU(gate) * up,
//   * q/k head RMSNorm + rotary embedding + K/V cache write + observation-window write, fused,
//   * the sampler's exponential race,
//   * the decode step's positions / context lengths / slots / window triples, on the device.
// All are streams over HBM with fp32 maths and the reference's rounding points (the value is
// rounded to the tensor dtype T wherever the reference's eager code holds it in a T tensor).
// IEEE division and square root are used where the reference divides or takes rsqrt, and
// products that the reference rounds separately are kept apart (__fmul_rn), so that fp32 results
// agree with it to the last bits of the reductions' summation order.
#include <type_traits>

#include "zp_common.cuh"

namespace zp {

// Two fp32 values rounded to T and back / stored as T, as one packed conversion where T is a
// 16-bit type (the scalar f32 -> 16-bit conversion issues at a quarter of the packed one's rate).
template <typename T> struct Two;
template <> struct Two<__nv_bfloat16> {
  static __device__ __forceinline__ void round(float& a, float& b) {
    const float2 f = __bfloat1622float2(__floats2bfloat162_rn(a, b));
    a = f.x; b = f.y;
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    p[0] = v.x; p[1] = v.y;
  }
};
template <> struct Two<__half> {
  static __device__ __forceinline__ void round(float& a, float& b) {
    const float2 f = __half22float2(__floats2half2_rn(a, b));
    a = f.x; b = f.y;
  }
  static __device__ __forceinline__ void store(__half* p, float a, float b) {
    const __half2 v = __floats2half2_rn(a, b);
    p[0] = v.x; p[1] = v.y;
  }
};
template <> struct Two<float> {
  static __device__ __forceinline__ void round(float&, float&) {}
  static __device__ __forceinline__ void store(float* p, float a, float b) { p[0] = a; p[1] = b; }
};

template <typename T> struct Vec16 {   // one 16-byte vector of T
  static constexpr int N = 16 / sizeof(T);
  int4 raw;
  __device__ __forceinline__ float get(int i) const { return Elem<T>::to_f32(reinterpret_cast<const T*>(&raw)[i]); }
  __device__ __forceinline__ void set(int i, float v) { reinterpret_cast<T*>(&raw)[i] = Elem<T>::from_f32(v); }
  __device__ __forceinline__ void set2(int i, float a, float b) { Two<T>::store(reinterpret_cast<T*>(&raw) + i, a, b); }
};

// ---------------------------------------------------------------------------------------------
// RMSNorm (+ residual).  One block per row; the row stays in registers between the two passes.
//   s = x (+ residual) in fp32;  residual_out = T(s);  y = T(T(s * rsqrt(mean(s^2) + eps)) * w)
// ---------------------------------------------------------------------------------------------
template <typename T, int VPT>
__global__ void __launch_bounds__(256)
rms_norm_kernel(const T* x, const T* residual, const T* weight,
                T* out, T* residual_out, int H, int64_t x_stride, int64_t out_stride, float eps) {
  __shared__ float red[32];
  constexpr int EPV = Vec16<T>::N;
  const int64_t row = blockIdx.x;
  const T* xr = x + row * x_stride;
  const T* rr = residual ? residual + row * (int64_t)H : nullptr;
  const int nvec = H / EPV;
  float s[VPT][EPV];
  float ss = 0.f;
  wait_for_previous();
  let_next_begin();
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + i * 256;
    if (v < nvec) {
      Vec16<T> a, b;
      a.raw = ld16(xr + v * EPV);
      if (rr) b.raw = ld16(rr + v * EPV);
#pragma unroll
      for (int j = 0; j < EPV; ++j) {
        s[i][j] = rr ? a.get(j) + b.get(j) : a.get(j);
        ss = fmaf(s[i][j], s[i][j], ss);
      }
      if (residual_out) {
        Vec16<T> o;
#pragma unroll
        for (int j = 0; j < EPV; j += 2) o.set2(j, s[i][j], s[i][j + 1]);
        st16(residual_out + row * (int64_t)H + v * EPV, o.raw);
      }
    }
  }
  ss = block_sum(ss, red);
  const float r = 1.f / sqrtf(ss / (float)H + eps);
  T* orow = out + row * out_stride;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + i * 256;
    if (v < nvec) {
      Vec16<T> w, o;
      w.raw = ld16(weight + v * EPV);
#pragma unroll
      for (int j = 0; j < EPV; j += 2) {
        float a = __fmul_rn(s[i][j], r), b = __fmul_rn(s[i][j + 1], r);
        Two<T>::round(a, b);
        o.set2(j, __fmul_rn(a, w.get(j)), __fmul_rn(b, w.get(j + 1)));
      }
      st16(orow + v * EPV, o.raw);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// out[n, i] = T( T(silu(x[n, i])) * x[n, I + i] ),  silu(a) = a / (1 + exp(-a)) in fp32
// ---------------------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ float silu_f32(float g) {
  // fp32 tensors: IEEE division and expf as the reference; 16-bit tensors: the fast forms' last-bit
  // errors disappear in the rounding to T (except at a rounding boundary, ~1 element in 10^4)
  if constexpr (sizeof(T) == 4) return g / (1.f + expf(-g));
  else return __fdividef(g, 1.f + __expf(-g));
}

// Bound by HBM: two vectors of each half a thread in flight, one block per 512 vectors; the row of a vector by a 32-bit division
// (`Index`) wherever the vectors can be counted in 32 bits: the 64-bit one took longer than the element's arithmetic.
// 8192 rows of 12288, bf16: 88 us = 6.9 TB/s (a grid-stride loop with 64-bit indices 119).
template <typename T, typename Index>
__global__ void __launch_bounds__(256)
silu_and_mul_kernel(const T* x, T* out, int I, Index total_vec) {
  wait_for_previous();
  let_next_begin();
  constexpr int EPV = Vec16<T>::N;
  const Index vec_per_row = I / EPV, v0 = (Index)blockIdx.x * 512 + threadIdx.x;
  Vec16<T> a[2], b[2];
  int64_t at[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {   // both loads of both vectors in flight before any maths
    const Index v = v0 + u * 256;
    if (v < total_vec) {
      const Index row = v / vec_per_row;
      const int64_t c = (int64_t)(v - row * vec_per_row) * EPV;
      at[u] = (int64_t)row * I + c;
      a[u].raw = ld16(x + (int64_t)row * 2 * I + c);
      b[u].raw = ld16(x + (int64_t)row * 2 * I + I + c);
    }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    if (v0 + u * 256 < total_vec) {
      Vec16<T> o;
#pragma unroll
      for (int j = 0; j < EPV; j += 2) {
        float s0 = silu_f32<T>(a[u].get(j)), s1 = silu_f32<T>(a[u].get(j + 1));
        Two<T>::round(s0, s1);
        o.set2(j, __fmul_rn(s0, b[u].get(j)), __fmul_rn(s1, b[u].get(j + 1)));
      }
      st16(out + at[u], o.raw);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Fused q/k RMSNorm + rotary embedding + cache writes.  A warp walks some heads of one kind (q, k or v) of one token, four at a
// time (eight lanes per head; a lane owns D/16 consecutive dims of each half of the head — the rotation pairs dim d with d + D/2
// — and moves them as one vector), with the next four heads' loads in flight: q heads -> q_out; k heads -> k_out and the K
// cache; v heads -> v_out (PACK: as attention over the rows themselves takes them) and the V cache, a plain copy.  Rows past the tokens
// redo the q heads of a window token and write them into the observation-window buffer.
//
// What bounds it is the loads in flight: with one kind of head a warp keeps one weight and the token's cosines and sines in
// registers (twice the warps per SM that a walk over all heads of a token left room for), and v heads do no arithmetic.  Many
// tokens: 32 heads a warp, so that cosines, sines and weights are fetched once for eight turns.  Few tokens (below QK_SPREAD,
// where a warp per token does not fill the SMs): four heads a warp, one turn of latency.
// 32 / 8 heads of 128, bf16: 16384 tokens 89 us = 4.9 TB/s (16 heads a warp 96, 8 105, 4 130; one warp for all kinds 114), 4 tokens
// 2.6 us (7.6).
//
// Registers (BLOCKS: of so many blocks an SM; 0: what the compiler takes for itself), heads of 128; those of 64 are the same either way.
// bf16 has 66 by itself and 79 of three blocks, which never lose: 4 tokens 1.72 -> 1.64 us, 2000 15.0 -> 13.5, 8192 43.5 -> 41.4, 12 prompts
// of 60 to 1500 tokens with packed values 54 -> 51 (54 for four blocks, 57 for five).  fp16 has 64 by itself, which is four blocks, or 78 of
// three: more registers are better while the blocks are no more than a wave or so (1100 tokens 12.1 -> 10.5, 1600 13.8 -> 11.1), more blocks
// from there on (1000 tokens in 1500 blocks 8.8 -> 9.5, 8192 38.7 -> 41.4).  fp32 has 90 by itself, two blocks, and spills a few
// in the 80 of three: 1100 tokens 12.1 -> 16.0, 4 tokens 1.70 -> 1.78, but 1000 12.9 -> 11.9 and 8192 68.8 -> 65.1.
// ---------------------------------------------------------------------------------------------
constexpr int QK_SPREAD = 1024;

struct QkArgs {
  const void* qkv; const int64_t* positions; const float* cos_sin;
  const void* q_weight; const void* k_weight;
  void* q_out; void* k_out; void* v_out; void* k_cache; void* v_cache;
  const int32_t* slot_mapping; void* query_cache; const int32_t* triples;
  const int32_t* n_triples_dev;   // NULL, or the device word that holds the number of valid triples
  int n_tokens, n_triples, Hq, Hkv;
  int64_t qkv_stride, cache_stride_seq, cache_stride_slot;
  float eps;
  int per, nq, nk;                // heads a warp walks; warps of a token's q heads, and of its k (and of its v) heads
};

// N consecutive elements of T moved as one (or two) vector accesses
template <typename T, int N>
struct alignas((sizeof(T) * N > 16) ? 16 : sizeof(T) * N) Chunk { T v[N]; };
template <typename T, int N>
__device__ __forceinline__ Chunk<T, N> ld_chunk(const T* p) { return *reinterpret_cast<const Chunk<T, N>*>(p); }
template <typename T, int N>
__device__ __forceinline__ void st_chunk(T* p, const Chunk<T, N>& c) { *reinterpret_cast<Chunk<T, N>*>(p) = c; }

// One head on its eight lanes: RMSNorm over the D dims (T(T(x * r) * w)), then the rotation in
// fp32 with separately rounded products, rounded to T once.  ca/cb: this lane's elements of the
// two halves of the head; w1/w2, c/s: its slices of the weight and of the token's cos/sin row.
template <typename T, int D>
__device__ __forceinline__ void norm_rope_head(const Chunk<T, D / 16>& ca, const Chunk<T, D / 16>& cb,
                                               const Chunk<T, D / 16>& w1, const Chunk<T, D / 16>& w2,
                                               const float (&c)[D / 16], const float (&s)[D / 16],
                                               float eps, Chunk<T, D / 16>& o1, Chunk<T, D / 16>& o2) {
  constexpr int P = D / 16;
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < P; ++j) {
    const float av = Elem<T>::to_f32(ca.v[j]), bv = Elem<T>::to_f32(cb.v[j]);
    ss = fmaf(av, av, ss);
    ss = fmaf(bv, bv, ss);
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);   // within the 8 lanes
  // fp32 tensors: IEEE square root and division as the reference's rsqrt; 16-bit tensors: the
  // fast reciprocal square root's last-bit error disappears in the rounding to T
  float r;
  if constexpr (sizeof(T) == 4) r = 1.f / sqrtf(ss / (float)D + eps);
  else r = rsqrtf(ss / (float)D + eps);
#pragma unroll
  for (int j = 0; j < P; j += 2) {
    // (the elements are unpacked again rather than kept in fp32 across the reduction: registers)
    float x1a = __fmul_rn(Elem<T>::to_f32(ca.v[j]), r), x1b = __fmul_rn(Elem<T>::to_f32(ca.v[j + 1]), r);
    float x2a = __fmul_rn(Elem<T>::to_f32(cb.v[j]), r), x2b = __fmul_rn(Elem<T>::to_f32(cb.v[j + 1]), r);
    Two<T>::round(x1a, x1b);
    Two<T>::round(x2a, x2b);
    x1a = __fmul_rn(x1a, Elem<T>::to_f32(w1.v[j])); x1b = __fmul_rn(x1b, Elem<T>::to_f32(w1.v[j + 1]));
    x2a = __fmul_rn(x2a, Elem<T>::to_f32(w2.v[j])); x2b = __fmul_rn(x2b, Elem<T>::to_f32(w2.v[j + 1]));
    Two<T>::round(x1a, x1b);
    Two<T>::round(x2a, x2b);
    Two<T>::store(o1.v + j, __fsub_rn(__fmul_rn(x1a, c[j]), __fmul_rn(x2a, s[j])),
                  __fsub_rn(__fmul_rn(x1b, c[j + 1]), __fmul_rn(x2b, s[j + 1])));
    Two<T>::store(o2.v + j, __fadd_rn(__fmul_rn(x2a, c[j]), __fmul_rn(x1a, s[j])),
                  __fadd_rn(__fmul_rn(x2b, c[j + 1]), __fmul_rn(x1b, s[j + 1])));
  }
}

template <typename T, int D, int BLOCKS, bool PACK>
__global__ void __launch_bounds__(256, BLOCKS) qk_norm_rope_store_kernel(const QkArgs a) {
  constexpr int P = D / 16;
  const int lane = threadIdx.x & 31, l8 = lane & 7, hg = lane >> 3;   // 4 heads per warp at a time
  const int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), part = blockIdx.y;
  const bool is_q = part < a.nq, is_v = part >= a.nq + a.nk, window = item >= a.n_tokens;
  wait_for_previous();
  let_next_begin();
  if (item >= a.n_tokens + a.n_triples || (window && !is_q)) return;
  int n = item, qid = 0, idx = 0;
  if (window) {
    const int t = item - a.n_tokens;
    if (a.n_triples_dev && t >= *a.n_triples_dev) return;   // n_triples was only the upper bound
    n = a.triples[3 * t]; qid = a.triples[3 * t + 1]; idx = a.triples[3 * t + 2];
  }
  const int heads = is_q ? a.Hq : a.Hkv, base = is_q ? 0 : is_v ? a.Hq + a.Hkv : a.Hq;   // of this kind, and where they start in a row
  const int h_begin = (part - (is_q ? 0 : is_v ? a.nq + a.nk : a.nq)) * a.per, h_end = min(h_begin + a.per, heads);
  const T* row = reinterpret_cast<const T*>(a.qkv) + (int64_t)n * a.qkv_stride + (int64_t)base * D;
  // the first heads' elements are requested before the (dependent) cos/sin loads
  auto load_head = [&](int h, Chunk<T, P>& ca, Chunk<T, P>& cb) {
    if (h < h_end) {
      ca = ld_chunk<T, P>(row + (int64_t)h * D + l8 * P);
      cb = ld_chunk<T, P>(row + (int64_t)h * D + D / 2 + l8 * P);
    } else {
#pragma unroll
      for (int j = 0; j < P; ++j) { ca.v[j] = Elem<T>::from_f32(0.f); cb.v[j] = Elem<T>::from_f32(0.f); }
    }
  };
  Chunk<T, P> ca, cb, na, nb;
  load_head(h_begin + hg, ca, cb);
  const int slot = !is_q && a.slot_mapping ? a.slot_mapping[n] : -1;
  if (is_v) {
    if constexpr (PACK) {
      T* d0 = reinterpret_cast<T*>(a.v_out) + (int64_t)n * a.Hkv * D;
      T* d1 = slot != -1 ? reinterpret_cast<T*>(a.v_cache) + (int64_t)slot * a.Hkv * D : nullptr;
      for (int h = h_begin + hg; h < h_end; h += 4) {
        load_head(h + 4, na, nb);
        const int64_t at = (int64_t)h * D + l8 * P;
        st_chunk<T, P>(d0 + at, ca); st_chunk<T, P>(d0 + at + D / 2, cb);
        if (d1) { st_chunk<T, P>(d1 + at, ca); st_chunk<T, P>(d1 + at + D / 2, cb); }
        ca = na; cb = nb;
      }
      return;
    }
    if (slot == -1) return;
    T* dst = reinterpret_cast<T*>(a.v_cache) + (int64_t)slot * a.Hkv * D;
    for (int h = h_begin + hg; h < h_end; h += 4) {
      load_head(h + 4, na, nb);
      st_chunk<T, P>(dst + (int64_t)h * D + l8 * P, ca);
      st_chunk<T, P>(dst + (int64_t)h * D + D / 2 + l8 * P, cb);
      ca = na; cb = nb;
    }
    return;
  }
  // this lane's slices of the token's cos/sin row and of the weight
  const float* cs = a.cos_sin + a.positions[n] * D;
  const T* wp = reinterpret_cast<const T*>(is_q ? a.q_weight : a.k_weight);
  float c[P], sn[P];
  {
    const Chunk<float, P> cc = ld_chunk<float, P>(cs + l8 * P), sc = ld_chunk<float, P>(cs + D / 2 + l8 * P);
#pragma unroll
    for (int j = 0; j < P; ++j) { c[j] = cc.v[j]; sn[j] = sc.v[j]; }
  }
  const Chunk<T, P> w1 = ld_chunk<T, P>(wp + l8 * P), w2 = ld_chunk<T, P>(wp + D / 2 + l8 * P);
  T* d0 = nullptr;                // where the heads go: output (or window buffer), ...
  T* d1 = nullptr;                // ... and cache
  if (window) d0 = reinterpret_cast<T*>(a.query_cache) + (int64_t)qid * a.cache_stride_seq + (int64_t)idx * a.cache_stride_slot;
  else if (is_q) d0 = reinterpret_cast<T*>(a.q_out) + (int64_t)n * a.Hq * D;
  else {
    if (a.k_out) d0 = reinterpret_cast<T*>(a.k_out) + (int64_t)n * a.Hkv * D;
    if (slot != -1) d1 = reinterpret_cast<T*>(a.k_cache) + (int64_t)slot * a.Hkv * D;
  }
  // every lane runs the same number of turns (the shuffles need the whole warp)
  for (int h0 = h_begin; h0 < h_end; h0 += 4) {
    const int h = h0 + hg;
    load_head(h + 4, na, nb);   // the next four heads, in flight while these are computed
    Chunk<T, P> o1, o2;
    norm_rope_head<T, D>(ca, cb, w1, w2, c, sn, a.eps, o1, o2);
    if (h < h_end) {
      const int64_t at = (int64_t)h * D + l8 * P;
      if (d0) { st_chunk<T, P>(d0 + at, o1); st_chunk<T, P>(d0 + at + D / 2, o2); }
      if (d1) { st_chunk<T, P>(d1 + at, o1); st_chunk<T, P>(d1 + at + D / 2, o2); }
    }
    ca = na; cb = nb;
  }
}

// ---------------------------------------------------------------------------------------------
// Sampler: probs = softmax(fp32 logits / T); token = argmax(probs / max(noise, 1e-10)), lowest
// index on ties.  A cluster of up to eight blocks per row, two passes over the row (the second from L2).  With
// noise == NULL the Exp(1) draws come from a counter-based generator keyed by (seed, row, index).
//
// What bounds it is arithmetic, some 25 instructions and, where every draw is made, three special-function operations per logit.
// A draw is at least the distance of its uniform number from 1, so an element can win only if that distance (the generator's
// bits, without a logarithm) is below e / the best ratio so far; the logarithm and the division are for the few that pass.
// Blocks of a row share its maximum, sum and best candidate through distributed shared memory: rows that leave SMs idle are spread
// over up to eight.  256 rows of 151936 bf16 logits: 65 us with one block a row (79 with four, 104 with eight; with all draws made, 1024
// threads and one block a row 105).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t mix32_upper(uint32_t x) {   // the upper 16 bits of mix32(x)
  x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu;
  return x;
}
__device__ __forceinline__ uint32_t mix32(uint32_t x) {   // a 32-bit finaliser (bijective)
  x = mix32_upper(x);
  return x ^ x >> 16;
}
__device__ __forceinline__ float exp1_draw(uint64_t seed, uint32_t row, uint32_t i) {
  uint32_t h = mix32(((uint32_t)seed ^ (row * 0x9e3779b9u)) + i * 0x85ebca6bu);
  h = mix32(h ^ (uint32_t)(seed >> 32) ^ row);
  const float u = ((float)(h >> 8) + 0.5f) * (1.0f / 16777216.0f);   // (0, 1)
  return -__logf(u);
}

constexpr int SAMPLE_SLICE = 6144, SAMPLE_SLICE_MANY = 32768;    // a row is spread over more blocks while each has this many logits

template <typename T, bool GIVEN, int SAMPLE_THREADS>      // GIVEN: the draws are given
__global__ void __launch_bounds__(SAMPLE_THREADS, SAMPLE_THREADS == 512 ? 3 : 1)
sample_kernel(const T* __restrict__ logits, const float* __restrict__ temperatures,
              const float* __restrict__ noise, int64_t* __restrict__ out, int V, int slice, uint64_t seed) {
  __shared__ float red[32], share_m, share_z, share_best;
  __shared__ int share_idx, bound;
  __shared__ float bval[32];
  __shared__ int bidx[32];
  const uint32_t rank = cluster_rank(), ranks = cluster_size();
  const int row = blockIdx.x / ranks;
  const T* lr = logits + (int64_t)row * V;
  const float t = temperatures[row];
  const int begin = min((int)rank * slice, V), end = min(begin + slice, V);
  // The block's part of the row in 16-byte vectors, and single elements before and behind them; a thread sees its
  // elements in ascending index order.  fn(first index, elements).
  constexpr int EPV = Vec16<T>::N;
  const int head = min((int)((16 - (uintptr_t)(lr + begin) % 16) % 16 / sizeof(T)), end - begin);
  const int nvec = (end - begin - head) / EPV, tail = begin + head + nvec * EPV;
  auto for_each = [&](auto deep, auto&& fn) {      // deep: vectors in flight
    if ((int)threadIdx.x < head) {
      const float x[1] = {Elem<T>::to_f32(lr[begin + threadIdx.x])};
      fn(begin + (int)threadIdx.x, x);
    }
    constexpr int N = decltype(deep)::value;
    for (int v0 = threadIdx.x; v0 < nvec; v0 += N * SAMPLE_THREADS) {
      Vec16<T> a[N];
#pragma unroll
      for (int u = 0; u < N; ++u)
        if (v0 + u * SAMPLE_THREADS < nvec) a[u].raw = ld16(lr + begin + head + (v0 + u * SAMPLE_THREADS) * EPV);
#pragma unroll
      for (int u = 0; u < N; ++u) {
        if (v0 + u * SAMPLE_THREADS >= nvec) break;
        float x[EPV];
#pragma unroll
        for (int j = 0; j < EPV; ++j) x[j] = a[u].get(j);
        fn(begin + head + (v0 + u * SAMPLE_THREADS) * EPV, x);
      }
    }
    for (int i = tail + threadIdx.x; i < end; i += SAMPLE_THREADS) {
      const float x[1] = {Elem<T>::to_f32(lr[i])};
      fn(i, x);
    }
  };
  auto row_max = [&](float m) -> float {      // over the block, then over the row's blocks
    m = block_max(m, red);
    if (ranks == 1) return m;
    if (threadIdx.x == 0) share_m = m;
    cluster_sync();
    for (uint32_t k = 0; k < ranks; ++k) m = fmaxf(m, ld_cluster(&share_m, k));
    cluster_sync();                           // (share_m may be rewritten)
    return m;
  };
  // Pass 1: the row maximum of logits / t.  For t > 0 the correctly rounded quotient is monotonic
  // in the numerator, so the maximum of the quotients is the quotient of the maximum.
  float mx = -INFINITY;
  using One = std::integral_constant<int, 1>;
  using Four = std::integral_constant<int, 4>;
  for_each(Four{}, [&](int, const auto& x) {
    for (float y : x) mx = fmaxf(mx, y);
  });
  mx = row_max(mx);
  float m = __fdiv_rn(mx, t);
  if (!(t > 0.f)) {   // a non-positive temperature: fall back to the literal maximum of the quotients
    m = -INFINITY;
    for_each(One{}, [&](int, const auto& x) {
      for (float y : x) m = fmaxf(m, __fdiv_rn(y, t));
    });
    m = row_max(m);
  }
  // Pass 2, with fast arithmetic: Z = sum of exp(x_i / t - m), and per thread the two best
  // candidates of the race e_i / q_i.  Dividing every e_i by Z (as the reference does) scales all
  // candidates alike, and the fast exp / reciprocal are off by a few units in the last place, so
  // only near-ties can be ordered differently by the reference's exact expression: the two best
  // per thread are re-evaluated with it below (correctly rounded divisions, expf), against the
  // same Z.
  // `bound`: a ratio that some element reaches; elements more than 2^-10 below it are left out.  At first the largest
  // element's, whose draw is at most -log(2^-25) < 17.4.
  const float inv_t = 1.f / t;
  if (threadIdx.x == 0) bound = __float_as_int(fmaxf(__expf(fmaf(mx, inv_t, -m)) * (1.f / 17.4f), 1e-30f));
  __syncthreads();
  float z = 0.f;
  float r0 = -INFINITY, r1 = -INFINITY, q0 = 1.f, q1 = 1.f;
  int i0 = 0x7fffffff, i1 = 0x7fffffff;
  auto race = [&](int i, float e) {
    const float q = fmaxf(GIVEN ? noise[(int64_t)row * V + i] : exp1_draw(seed, row, i), 1e-10f);
    const float r = __fdividef(e, q);
    if (r > r1) {
      if (r > r0) { r1 = r0; q1 = q0; i1 = i0; r0 = r; q0 = q; i0 = i; }
      else { r1 = r; q1 = q; i1 = i; }
      if constexpr (!GIVEN)
        if (__float_as_int(r) > *(volatile int*)&bound) atomicMax(&bound, __float_as_int(r));      // (r >= 0: ordered as its bits)
    }
  };
  const uint32_t hash0 = (uint32_t)seed ^ ((uint32_t)row * 0x9e3779b9u), hash1 = (uint32_t)(seed >> 32) ^ (uint32_t)row;
  for_each(One{}, [&](int first, const auto& x) {
    constexpr int n = sizeof(x) / sizeof(float);
    float e[n];
#pragma unroll
    for (int j = 0; j < n; ++j) {
      e[j] = __expf(fmaf(x[j], inv_t, -m));
      z += e[j];
    }
    if constexpr (GIVEN) {
#pragma unroll
      for (int j = 0; j < n; ++j) race(first + j, e[j]);
    } else {
      // e / best >= 1 - u, in units of 2^-23: the generator's upper bits, inverted, as the mantissa of a number from 2^23 on.  Its
      // last step changes the lower half of its bits alone, so the test leaves that step out and allows for 2^-16 (128 units), and
      // for the rounding of u and the error of the fast logarithm (ten)
      const float per = __fdividef(8388608.f * 1.001f, __int_as_float(*(volatile int*)&bound));
      float over = -1.f;
      float d[n];
#pragma unroll
      for (int j = 0; j < n; ++j) {
        const uint32_t h = mix32_upper(mix32(hash0 + (uint32_t)(first + j) * 0x85ebca6bu) ^ hash1);
        d[j] = fmaf(e[j], per, 8388608.f + 138.f - __uint_as_float((~h >> 9) | 0x4b000000u));
        over = fmaxf(over, d[j]);
      }
      if (over >= 0.f) {
#pragma unroll
        for (int j = 0; j < n; ++j)
          if (d[j] >= 0.f) race(first + j, e[j]);
      }
    }
  });
  z = block_sum(z, red);
  if (ranks > 1) {
    if (threadIdx.x == 0) share_z = z;
    cluster_sync();
    z = 0.f;
    for (uint32_t k = 0; k < ranks; ++k) z += ld_cluster(&share_z, k);
  }
  // the reference's value of a candidate: (exp(x / t - m) / Z) / q
  auto exact = [&](int i, float q) -> float {
    if (i == 0x7fffffff) return -INFINITY;
    const float e = expf(__fdiv_rn(Elem<T>::to_f32(lr[i]), t) - m);
    return __fdiv_rn(__fdiv_rn(e, z), q);
  };
  const float v0 = exact(i0, q0), v1 = exact(i1, q1);
  float best = v0;
  int besti = i0;
  if (v1 > best || (v1 == best && i1 < besti)) { best = v1; besti = i1; }
  // (value, index) arg-max: larger value wins, then the lower index
  auto warp_best = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, besti, o);
      if (ov > best || (ov == best && oi < besti)) { best = ov; besti = oi; }
    }
  };
  warp_best();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = SAMPLE_THREADS >> 5;
  if (lane == 0) { bval[w] = best; bidx[w] = besti; }
  __syncthreads();
  if (w == 0) {
    best = lane < nw ? bval[lane] : -INFINITY;
    besti = lane < nw ? bidx[lane] : 0x7fffffff;
    warp_best();
    if (lane == 0) { share_best = best; share_idx = besti; }
  }
  if (ranks > 1) {
    cluster_sync();
    if (rank == 0 && w == 0) {
      best = lane < (int)ranks ? ld_cluster(&share_best, lane) : -INFINITY;
      besti = lane < (int)ranks ? __float_as_int(ld_cluster(reinterpret_cast<const float*>(&share_idx), lane)) : 0x7fffffff;
      warp_best();
    }
    cluster_sync();    // (a block's shared memory stays until the others have read it)
  }
  if (rank == 0 && threadIdx.x == 0) out[row] = besti == 0x7fffffff ? 0 : besti;      // (no number in the row is above zero: any token)
}

template <typename T>
static int launch_sample(const T* logits, const float* temperatures, const float* noise, int64_t* out, int rows, int V, uint64_t seed, cudaStream_t st) {
  // Blocks of a row meet four times, which costs more than an even load gains unless SMs idle and a row is long.
  // 151936 logits, 1, 2, 4, 8 blocks a row (us): 1 row 40, 27, 18, 15; 37: 41, 28, 28, 26; 55: 42, 29, 29, 36; 74: 42, 30, 37, 43; 90: 43, 43, 37, 50; 110: 44,
  // 44, 49, 58; 222: 74, 64, 83, 105; 300: 103, 95, 101, 138.  32000: 1 row 14, 13, 12, 11; 74: 15, 15, 18, 27; 110: 15, 18, 24, 35.
  // Given draws are loads: a block of 1024 threads where a row has an SM to itself.  151936 fp32 logits: 1 row 36, 26, 18, 15; 16: 37, 27, 20, 28; 37: 37, 28, 35,
  // 42; 74: 43, 33, 54, 72; 110: 50, 60, 76, 114.
  const bool wide = noise && rows <= 148;
  const int most = wide ? (rows <= 12 ? 8 : rows <= 27 ? 4 : rows <= 74 ? 2 : 1) : rows <= 37 ? 8 : rows <= 100 ? 4 : rows <= 222 ? 2 : 1;
  const int part = rows <= 74 ? SAMPLE_SLICE : SAMPLE_SLICE_MANY;
  int ranks = 1;
  while (ranks < most && V / (2 * ranks) >= part) ranks *= 2;
  const int slice = ((V + ranks - 1) / ranks + 63) / 64 * 64;
  auto run = [&](auto kernel, int threads) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)rows * ranks);
    cfg.blockDim = dim3(threads);
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = ranks; attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = ranks > 1;      // (a block alone is a cluster as it is)
    return cudaLaunchKernelEx(&cfg, kernel, logits, temperatures, noise, out, V, slice, seed);
  };
  const cudaError_t e = !noise ? run(sample_kernel<T, false, 512>, 512) : wide ? run(sample_kernel<T, true, 1024>, 1024) : run(sample_kernel<T, true, 512>, 512);
  if (e != cudaSuccess) { set_error("zp_sample: %s", cudaGetErrorString(e)); return ZP_ERR_CUDA; }
  return check_launch("zp_sample");
}

// A decode step's inputs into the buffers that a graph reads; rows and columns past the live ones are cleared.  Bound by the launch:
// one instead of four copies and, for a batch that is not full, three fills (about 2 us each on the device).
__global__ void __launch_bounds__(64)
decode_inputs_kernel(const int64_t* ids, const int32_t* num, const int32_t* tab, int64_t tab_stride, const int32_t* qid, int n, int width,
                     int64_t* ids_out, int32_t* num_out, int32_t* tab_out, int32_t* qid_out, int max_width) {
  const int row = blockIdx.x;
  const bool live = row < n;
  for (int c = threadIdx.x; c < max_width; c += 64)
    tab_out[(int64_t)row * max_width + c] = live && c < width ? tab[row * tab_stride + c] : -1;
  if (threadIdx.x == 0) {
    num_out[row] = live ? num[row] : 0;
    qid_out[row] = live ? qid[row] : -1;
    if (live) ids_out[row] = ids[row];
  }
}

// ---------------------------------------------------------------------------------------------
// Decode bookkeeping from device-resident state.  One block; the window triples keep the order
// of the sequences (block-wide exclusive scan of the "has a triple" flags).
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(1024)
prepare_decode_kernel(const int32_t* __restrict__ num_tokens, const int32_t* __restrict__ block_tables,
                      const int32_t* __restrict__ query_ids, int B, int W, int qcl, int bs,
                      int64_t* __restrict__ positions, int32_t* __restrict__ context_lens,
                      int32_t* __restrict__ slot_mapping, int32_t* __restrict__ triples,
                      int32_t* __restrict__ n_triples) {
  __shared__ int wsum[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int base = 0; base < B; base += blockDim.x) {
    const int i = base + threadIdx.x;
    int flag = 0, qid = -1, widx = 0;
    if (i < B) {
      const int n = num_tokens[i];
      const int nblocks = (n + bs - 1) / bs;
      const int last = n - (nblocks - 1) * bs;          // tokens in the last page, 1..bs
      int len = 0;
      while (len < W && block_tables[(int64_t)i * W + len] != -1) ++len;
      const int last_page = len > 0 ? block_tables[(int64_t)i * W + len - 1] : 0;
      if (n > 0 && len > 0) {
        positions[i] = n - 1;
        context_lens[i] = (len - 1) * bs + last;
        slot_mapping[i] = last_page * bs + last - 1;
        qid = query_ids[i];
        flag = qid != -1 && last > bs - qcl;
        widx = last - (bs - qcl) - 1;
      } else {  // a padding row of a fixed-size (graph) batch: nothing is stored, nothing attended
        positions[i] = 0;
        context_lens[i] = 0;
        slot_mapping[i] = -1;
      }
    }
    // exclusive scan of `flag` over the block
    int incl = flag;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    if (w == 0) {
      int s = lane < nw ? wsum[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += v;
      }
      wsum[lane] = s;   // inclusive over warps
    }
    __syncthreads();
    const int before = carry + (w > 0 ? wsum[w - 1] : 0) + incl - flag;
    if (flag) {
      triples[3 * before] = i;
      triples[3 * before + 1] = qid;
      triples[3 * before + 2] = widx;
    }
    __syncthreads();
    if (threadIdx.x == 0) carry += wsum[nw - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0) *n_triples = carry;
}

}  // namespace zp

extern "C" int zp_rms_norm(const void* x, const void* residual, const void* weight, void* out,
                           void* residual_out, int n_rows, int hidden, int64_t x_stride,
                           int64_t out_stride, float eps, int dtype, void* stream) {
  if (n_rows == 0) return ZP_OK;
  ZP_REQUIRE(x && weight && out, "zp_rms_norm: null pointer");
  ZP_REQUIRE(!residual_out || residual, "zp_rms_norm: residual_out without residual");
  const size_t es = zp::dtype_size(dtype);
  const int epv = (int)(16 / es);
  ZP_REQUIRE(hidden % epv == 0 && (x_stride * es) % 16 == 0 && (out_stride * es) % 16 == 0,
             "zp_rms_norm: rows must be multiples of 16 bytes");
  ZP_REQUIRE(((uintptr_t)x | (uintptr_t)residual | (uintptr_t)weight | (uintptr_t)out |
              (uintptr_t)residual_out) % 16 == 0, "zp_rms_norm: pointers must be 16-byte aligned");
  const int nvec = hidden / epv;
  ZP_REQUIRE(nvec <= 256 * 8, "zp_rms_norm: hidden size %d too large (at most %d)", hidden, 256 * 8 * epv);
  cudaStream_t st = (cudaStream_t)stream;
  ZP_DISPATCH_DTYPE(dtype, T, {
    const T* xp = (const T*)x; const T* rp = (const T*)residual; const T* wp = (const T*)weight;
    T* op = (T*)out; T* rop = (T*)residual_out;
    if (nvec <= 256) zp::launch_early(zp::rms_norm_kernel<T, 1>, dim3(n_rows), 256, 0, st, xp, rp, wp, op, rop, hidden, x_stride, out_stride, eps);
    else if (nvec <= 512) zp::launch_early(zp::rms_norm_kernel<T, 2>, dim3(n_rows), 256, 0, st, xp, rp, wp, op, rop, hidden, x_stride, out_stride, eps);
    else if (nvec <= 1024) zp::launch_early(zp::rms_norm_kernel<T, 4>, dim3(n_rows), 256, 0, st, xp, rp, wp, op, rop, hidden, x_stride, out_stride, eps);
    else zp::launch_early(zp::rms_norm_kernel<T, 8>, dim3(n_rows), 256, 0, st, xp, rp, wp, op, rop, hidden, x_stride, out_stride, eps);
  });
  return zp::check_launch("zp_rms_norm");
}

extern "C" int zp_silu_and_mul(const void* x, void* out, int n_rows, int inter, int dtype, void* stream) {
  if (n_rows == 0 || inter == 0) return ZP_OK;
  ZP_REQUIRE(x && out, "zp_silu_and_mul: null pointer");
  const size_t es = zp::dtype_size(dtype);
  const int epv = (int)(16 / es);
  ZP_REQUIRE(inter % epv == 0, "zp_silu_and_mul: the intermediate size must be a multiple of %d", epv);
  ZP_REQUIRE(((uintptr_t)x | (uintptr_t)out) % 16 == 0, "zp_silu_and_mul: pointers must be 16-byte aligned");
  const int64_t total_vec = (int64_t)n_rows * (inter / epv);
  const int64_t blocks = (total_vec + 511) / 512;
  ZP_REQUIRE(blocks <= 0x7fffffff, "zp_silu_and_mul: too many rows");
  ZP_DISPATCH_DTYPE(dtype, T, {
    if (total_vec < (1ll << 31))
      zp::launch_early(zp::silu_and_mul_kernel<T, uint32_t>, dim3((unsigned)blocks), 256, 0, (cudaStream_t)stream, (const T*)x, (T*)out, inter, (uint32_t)total_vec);
    else
      zp::launch_early(zp::silu_and_mul_kernel<T, int64_t>, dim3((unsigned)blocks), 256, 0, (cudaStream_t)stream, (const T*)x, (T*)out, inter, total_vec);
  });
  return zp::check_launch("zp_silu_and_mul");
}

extern "C" int zp_qk_norm_rope_store_v(const void* qkv, const int64_t* positions, const float* cos_sin,
                                     const void* q_weight, const void* k_weight, float eps,
                                     void* q_out, void* k_out, void* v_out, void* k_cache, void* v_cache,
                                     const int32_t* slot_mapping, void* query_cache,
                                     const int32_t* triples, int n_triples,
                                     const int32_t* n_triples_device, int n_tokens, int Hq,
                                     int Hkv, int D, int64_t qkv_stride, int64_t cache_stride_seq,
                                     int64_t cache_stride_slot, int dtype, void* stream) {
  if (n_tokens == 0) return ZP_OK;
  ZP_REQUIRE(qkv && positions && cos_sin && q_weight && k_weight && q_out, "zp_qk_norm_rope_store: null pointer");
  ZP_REQUIRE(!slot_mapping || (k_cache && v_cache), "zp_qk_norm_rope_store: slot mapping without caches");
  ZP_REQUIRE(n_triples == 0 || (triples && query_cache), "zp_qk_norm_rope_store: window triples without a buffer");
  ZP_REQUIRE(D == 64 || D == 128, "zp_qk_norm_rope_store: head_dim %d not supported (64 or 128)", D);
  {
    const size_t es = zp::dtype_size(dtype);
    const size_t vec = (D / 16) * es > 16 ? 16 : (D / 16) * es;   // the widest vector access used
    ZP_REQUIRE(((uintptr_t)qkv | (uintptr_t)q_weight | (uintptr_t)k_weight | (uintptr_t)q_out |
                (uintptr_t)k_out | (uintptr_t)v_out | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)query_cache |
                (uintptr_t)cos_sin) % 16 == 0 && (qkv_stride * es) % vec == 0 &&
                   (cache_stride_seq * es) % vec == 0 && (cache_stride_slot * es) % vec == 0,
               "zp_qk_norm_rope_store: pointers must be 16-byte aligned and strides vector-aligned");
  }
  zp::QkArgs a;
  a.qkv = qkv; a.positions = positions; a.cos_sin = cos_sin; a.q_weight = q_weight; a.k_weight = k_weight;
  a.q_out = q_out; a.k_out = k_out; a.v_out = v_out; a.k_cache = k_cache; a.v_cache = v_cache;
  a.slot_mapping = slot_mapping; a.query_cache = query_cache; a.triples = triples;
  a.n_triples_dev = n_triples_device;
  a.n_tokens = n_tokens; a.n_triples = n_triples; a.Hq = Hq; a.Hkv = Hkv;
  a.qkv_stride = qkv_stride; a.cache_stride_seq = cache_stride_seq; a.cache_stride_slot = cache_stride_slot;
  a.eps = eps;
  cudaStream_t st = (cudaStream_t)stream;
  a.per = n_tokens < zp::QK_SPREAD ? 4 : 32;
  a.nq = (Hq + a.per - 1) / a.per;
  a.nk = (Hkv + a.per - 1) / a.per;
  const dim3 grid((n_tokens + n_triples + 7) / 8, a.nq + 2 * a.nk);   // eight warps per block, one token each
  ZP_DISPATCH_DTYPE(dtype, T, {
    constexpr bool bf16 = std::is_same<T, __nv_bfloat16>::value;
    const int64_t blocks = (int64_t)grid.x * grid.y;
    const bool three = bf16 || (std::is_same<T, float>::value ? blocks > 4 * 148 : blocks <= 5 * 148);
    auto go = [&](auto pack) {
      constexpr bool PACK = decltype(pack)::value;
      if (D == 64) zp::launch_early(zp::qk_norm_rope_store_kernel<T, 64, 3, PACK>, grid, 256, 0, st, a);
      else if (three) zp::launch_early(zp::qk_norm_rope_store_kernel<T, 128, 3, PACK>, grid, 256, 0, st, a);
      else zp::launch_early(zp::qk_norm_rope_store_kernel<T, 128, bf16 ? 3 : 0, PACK>, grid, 256, 0, st, a);
    };
    if (v_out) go(std::true_type());
    else go(std::false_type());
  });
  return zp::check_launch("zp_qk_norm_rope_store");
}

extern "C" int zp_qk_norm_rope_store(const void* qkv, const int64_t* positions, const float* cos_sin,
                                     const void* q_weight, const void* k_weight, float eps,
                                     void* q_out, void* k_out, void* k_cache, void* v_cache,
                                     const int32_t* slot_mapping, void* query_cache,
                                     const int32_t* triples, int n_triples,
                                     const int32_t* n_triples_device, int n_tokens, int Hq,
                                     int Hkv, int D, int64_t qkv_stride, int64_t cache_stride_seq,
                                     int64_t cache_stride_slot, int dtype, void* stream) {
  return zp_qk_norm_rope_store_v(qkv, positions, cos_sin, q_weight, k_weight, eps, q_out, k_out, nullptr, k_cache, v_cache, slot_mapping, query_cache,
                                 triples, n_triples, n_triples_device, n_tokens, Hq, Hkv, D, qkv_stride, cache_stride_seq, cache_stride_slot, dtype, stream);
}

extern "C" int zp_sample(const void* logits, const float* temperatures, const float* noise,
                         int64_t* tokens_out, int n_rows, int vocab, uint64_t seed, int dtype,
                         void* stream) {
  if (n_rows == 0) return ZP_OK;
  ZP_REQUIRE(logits && temperatures && tokens_out, "zp_sample: null pointer");
  ZP_REQUIRE(vocab > 0, "zp_sample: empty vocabulary");
  ZP_DISPATCH_DTYPE(dtype, T, {
    return zp::launch_sample<T>((const T*)logits, temperatures, noise, tokens_out, n_rows, vocab, seed, (cudaStream_t)stream);
  });
  return ZP_OK;
}

extern "C" int zp_decode_inputs(const int64_t* input_ids, const int32_t* num_tokens, const int32_t* block_tables, int64_t table_stride,
                                const int32_t* query_ids, int n, int width, int64_t* input_ids_out, int32_t* num_tokens_out,
                                int32_t* block_tables_out, int32_t* query_ids_out, int max_n, int max_width, void* stream) {
  if (max_n == 0) return ZP_OK;
  ZP_REQUIRE(n >= 0 && n <= max_n && width >= 0 && width <= max_width, "zp_decode_inputs: more rows or columns than the buffers have");
  ZP_REQUIRE(input_ids_out && num_tokens_out && block_tables_out && query_ids_out && (n == 0 || (input_ids && num_tokens && query_ids)) &&
                 (n == 0 || width == 0 || block_tables), "zp_decode_inputs: null pointer");
  zp::decode_inputs_kernel<<<max_n, 64, 0, (cudaStream_t)stream>>>(input_ids, num_tokens, block_tables, table_stride, query_ids, n, width,
                                                                   input_ids_out, num_tokens_out, block_tables_out, query_ids_out, max_width);
  return zp::check_launch("zp_decode_inputs");
}

extern "C" int zp_prepare_decode(const int32_t* num_tokens, const int32_t* block_tables,
                                 const int32_t* query_ids, int B, int table_width,
                                 int query_cache_len, int block_size, int64_t* positions_out,
                                 int32_t* context_lens_out, int32_t* slot_mapping_out,
                                 int32_t* triples_out, int32_t* n_triples_out, void* stream) {
  ZP_REQUIRE(n_triples_out, "zp_prepare_decode: null pointer");
  if (B == 0) return cudaMemsetAsync(n_triples_out, 0, sizeof(int32_t), (cudaStream_t)stream) == cudaSuccess
                         ? ZP_OK : ZP_ERR_CUDA;
  ZP_REQUIRE(num_tokens && block_tables && query_ids && positions_out && context_lens_out &&
                 slot_mapping_out && triples_out, "zp_prepare_decode: null pointer");
  ZP_REQUIRE(table_width > 0 && block_size > 0 && query_cache_len >= 0 && query_cache_len <= block_size,
             "zp_prepare_decode: bad sizes");
  zp::prepare_decode_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(
      num_tokens, block_tables, query_ids, B, table_width, query_cache_len, block_size, positions_out,
      context_lens_out, slot_mapping_out, triples_out, n_triples_out);
  return zp::check_launch("zp_prepare_decode");
}

// Variable-length causal prefill attention (bottom-right aligned) on tcgen05 tensor cores: 16-bit tensors, head_dim 128,
// K/V dense or paged (page size a multiple of 128).  The pipeline is the one of zp_attn_tc.cuh; the weights enter the
// second product as T, as in the reference's attention.
//
// A work item is two heads of one key/value head over the same 128 queries, so that a key tile is fetched once for
// both; where a key/value head has an odd number of heads it is two neighbouring query tiles of one head.
//
// One group of softmax warps a tile, which hands over its first 64 weights behind half of the second 64's exponentials (the store
// is over by then: 1 x 16384 tokens 2.30 -> 2.26 ms a call); two for single tiles of up to four key tiles.  The second group's earlier
// start is the gain, the exchange of every step's maximum the price.  Kernel alone, one group / two (us): prompts of 40 tokens 10.4 / 10.0,
// 300 14.5 / 14.3, 400 16.8 / 16.6, 8 of 40 11.1 / 10.7; 700 20.5 / 21.0, 1500 31.6 / 33.1, 2000 (8 heads) 39.4 / 41.5; behind 256 cached keys
// 40 tokens 14.5 / 14.5, 200 16.2 / 16.6, 700 23.9 / 24.7; behind 1024 40 tokens 26.0 / 26.8.
//
// Measured (32 / 8 heads, bf16; causal count), single calls and SM clock: 1 x 16384 tokens 2.0 ms at 1.83 GHz = 1100 TFLOP/s, 2.25 ms at the
// 1.62 GHz that are left after some dozens of them (power), 4 x 4096 0.63 ms, 12 prompts of 60 to 1500 tokens 150 us. One query tile a block with a
// pass for the row maxima and one for the weights: 3.46 ms at 1.78 GHz, 1.09 ms, 282 us at 1.96 GHz.
#include "zp_attn_tc.cuh"

namespace zp {

using namespace attn;

template <typename T_, int GROUPS_> struct PrefillTc {
  using T = T_;
  static constexpr bool SPLIT = false, MASKED = false, CAPPED = false, BIASED = false, GATED = false;
  static constexpr int GROUPS = GROUPS_;
  // weights up to 2^LAZY: bf16 has fp32's range; fp16 ends at 2^16
  static constexpr float LAZY = UmmaFmt<T>::fmt == 1 ? 40.f : 12.f;
  CUtensorMap tmQ, tmK, tmV;
  const int32_t *cu_q, *cu_k, *table;
  void* o;
  int* error_word;
  Rings rings;
  int NBmax, Hq, Hkv, BS, levels, dv, mode;
  float scale_log2e;

  __device__ __forceinline__ void prefetch() const {
    prefetch_tensormap(&tmQ);
    prefetch_tensormap(&tmK);
    prefetch_tensormap(&tmV);
  }
  __device__ __forceinline__ bool item(dim3 id, Item& it) const {
    const int b = id.y, level = levels - 1 - (int)id.z;
    const int q0 = cu_q[b], lq = cu_q[b + 1] - q0, lk = cu_k[b + 1] - cu_k[b];
    const int first = level * level_rows(mode);
    if (first >= lq) return false;
    it.b = b;
    it.keys = lk;
    it.kept = it.t0 = 0;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int qi = item_row(mode, first, t), rows = item_rows(mode, lq - qi, t);
      it.head[t] = item_head(mode, id.x, t);
      it.q0[t] = q0 + qi;
      it.rows[t] = rows;
      it.pos[t] = qi + lk - lq;
      const int seen = rows > 0 ? min(lk, it.pos[t] + rows) : 0;      // keys that any row of the tile sees
      it.n[t] = seen > 0 ? (seen + 127) >> 7 : 0;
    }
    it.hk = it.head[0] / (Hq / Hkv);
    return true;
  }
  __device__ __forceinline__ void load_q(unsigned char* dst, uint64_t* bar, const Item& it, int t) const {
    for (int i = 0; i < 2; ++i) tma_load_5d(dst + i * BLK, &tmQ, bar, i * 64, it.head[t], it.q0[t], 0, 0);
  }
  struct Step {
    int row, page;
    __device__ __forceinline__ Step(const PrefillTc& p, const Item& it, int key0)
        : row(p.table ? key0 % p.BS : p.cu_k[it.b] + key0), page(p.table ? p.table[(int64_t)it.b * p.NBmax + key0 / p.BS] : 0) {}
  };
  __device__ __forceinline__ void load_k(unsigned char* dst, uint64_t* bar, const Item& it, const Step& s, int i) const {
    tma_load_5d(dst, &tmK, bar, i * 64, it.hk, s.row, s.page, 0);
  }
  __device__ __forceinline__ void load_v(unsigned char* dst, uint64_t* bar, const Item& it, const Step& s, int i) const {
    tma_load_5d(dst, &tmV, bar, i * 64, it.hk, s.row, s.page, 0);
  }
  __device__ __forceinline__ T* out(int row, int head, int c) const { return reinterpret_cast<T*>(o) + ((int64_t)row * Hq + head) * 128 + c; }

  struct Row {
    int lim;
    float ref0;
    Factor fac;
    __device__ __forceinline__ Row(const PrefillTc& p, const Item& it, int t, int r)
        : lim(min(it.keys - 1, of_tile(it.pos, t) + r)), ref0(-INFINITY), fac(p.scale_log2e) {}
    __device__ __forceinline__ float finish(const PrefillTc&, float, float l) const { return l > 0.f ? 1.f / l : 0.f; }
  };
};

template <typename T, int GROUPS>
static int launch_prefill_tc(const void* q, const void* k, const void* v, PrefillTc<T, GROUPS>& p, int B, int max_seqlen_q,
                             int64_t kv_stride_page, int total_q, int total_k, cudaStream_t st) {
  const uint32_t box[5] = {64, 1, 128, 1, 1};
  {
    const uint64_t dims[5] = {128, (uint64_t)p.Hq, (uint64_t)total_q, 1, 1};
    const uint64_t strides[4] = {128, (uint64_t)p.Hq * 128, (uint64_t)p.Hq * 128, (uint64_t)p.Hq * 128};
    if (int rc = make_tensor_map_5d(&p.tmQ, UmmaFmt<T>::tm, q, dims, strides, box, sizeof(T))) return rc;
  }
  const uint64_t row = (uint64_t)p.Hkv * 128, page = p.table ? (uint64_t)kv_stride_page : row;
  const uint64_t dims[5] = {128, (uint64_t)p.Hkv, (uint64_t)(p.table ? p.BS : total_k), p.table ? 1ull << 30 : 1ull, 1};
  const uint64_t strides[4] = {128, row, page, page};
  if (int rc = make_tensor_map_5d(&p.tmK, UmmaFmt<T>::tm, k, dims, strides, box, sizeof(T))) return rc;
  if (int rc = make_tensor_map_5d(&p.tmV, UmmaFmt<T>::tm, v, dims, strides, box, sizeof(T))) return rc;
  p.rings = rings_of(2, 2);
  p.dv = 128;
  const dim3 grid = grid_of(p.mode, p.Hq, B, max_seqlen_q, p.levels);
  return launch_attn(p, grid, st, "zp_varlen_prefill(tcgen05)");
}

// Called by zp_varlen_prefill_ex (zp_prefill.cu).
// total_q / total_k: rows of q and (dense case) of k and v (tensor-map extents: rows past them read as 0).
int varlen_prefill_tc(const void* q, const void* k, const void* v, const int32_t* cu_q, const int32_t* cu_k,
                      const int32_t* table, void* out, int B, int max_seqlen_q, int NBmax, int Hq, int Hkv,
                      int BS, int64_t kv_stride_page, float scale_log2e, int total_q, int total_k, int dtype,
                      cudaStream_t st) {
  const int mode = pick_mode(Hq, Hq / Hkv, B, total_q, max_seqlen_q);
  auto run = [&](auto p) {
    p.cu_q = cu_q; p.cu_k = cu_k; p.table = table; p.o = out;
    p.error_word = device_error_word();
    p.mode = mode;
    p.NBmax = NBmax; p.Hq = Hq; p.Hkv = Hkv; p.BS = BS; p.scale_log2e = scale_log2e;
    if (!p.error_word) { set_error("zp_varlen_prefill(tcgen05): no device error word"); return (int)ZP_ERR_CUDA; }
    return launch_prefill_tc(q, k, v, p, B, max_seqlen_q, kv_stride_page, total_q, total_k, st);
  };
  const bool two = mode == SINGLE && !table && max_seqlen_q <= 512 && total_k <= total_q;      // groups of softmax warps
  if (dtype == ZP_DTYPE_BF16) return two ? run(PrefillTc<__nv_bfloat16, 2>{}) : run(PrefillTc<__nv_bfloat16, 1>{});
  if (dtype == ZP_DTYPE_F16) return two ? run(PrefillTc<__half, 2>{}) : run(PrefillTc<__half, 1>{});
  set_error("zp_varlen_prefill(tcgen05): 16-bit tensors only");
  return ZP_ERR_UNSUPPORTED;
}

}  // namespace zp

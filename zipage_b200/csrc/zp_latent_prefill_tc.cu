// Causal attention of prompt portions over keys and values computed from latents, on tcgen05 tensor cores
// (bf16): a key is an unrotated part of its head's own and a rotated part that all heads share, so the two are
// fetched from where they lie (the expanded keys, the latent rows) and meet only in the accumulator:
//   S = Qn Kn^T + Qr Kr^T       [128 queries, 128 keys]
// The pipeline is the one of zp_attn_tc.cuh, with the weights as bf16 hi + lo.  A work item is two neighbouring query tiles
// of one head (every head has keys and values of its own).  Parts whose sizes are not multiples of 64 are filled with
// zeros by TMA.
//
// A tile of its own per block, all softmax warps on it, left the tensor cores idle during each of its softmax turns.  Three portions of
// 600 to 3000 tokens, 32 heads of 128 + 64: 309 to 337 us (460 so); with two groups of softmax warps a tile 6 us less.
#include "zp_attn_tc.cuh"
#include "zp_latent.cuh"

namespace zp {

using namespace attn;

struct LatentPrefillTc {
  using T = __nv_bfloat16;
  static constexpr bool SPLIT = true, MASKED = false, CAPPED = false, BIASED = false, GATED = false;
  static constexpr int GROUPS = 2;
  static constexpr float LAZY = 40.f;
  CUtensorMap tmQn, tmQr, tmKn, tmKr, tmV;
  const int32_t *cu_q, *cu_k;
  T* o;
  int* error_word;
  Rings rings;
  int nbn, levels, dv, mode; // 64-entry blocks of the unrotated part
  int64_t out_stride;
  float scale_log2e;

  __device__ __forceinline__ void prefetch() const {
    prefetch_tensormap(&tmQn);
    prefetch_tensormap(&tmQr);
    prefetch_tensormap(&tmKn);
    prefetch_tensormap(&tmKr);
    prefetch_tensormap(&tmV);
  }
  __device__ __forceinline__ bool item(dim3 id, Item& it) const {
    const int b = id.y, first = (levels - 1 - (int)id.z) * level_rows(mode);
    const int q0 = cu_q[b], lq = cu_q[b + 1] - q0, lk = cu_k[b + 1] - cu_k[b];
    if (first >= lq || lk < lq) return false;
    it.b = b;
    it.hk = id.x;
    it.keys = lk;
    it.kept = it.t0 = 0;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int qi = item_row(mode, first, t);
      it.head[t] = id.x;
      it.q0[t] = q0 + qi;
      it.rows[t] = item_rows(mode, lq - qi, t);
      it.pos[t] = qi + lk - lq;
      it.n[t] = it.rows[t] > 0 ? ((it.pos[t] + it.rows[t] - 1) >> 7) + 1 : 0;
    }
    return true;
  }
  __device__ __forceinline__ void load_q(unsigned char* dst, uint64_t* bar, const Item& it, int t) const {
    for (int i = 0; i < rings.nbq; ++i)
      tma_load_5d(dst + i * BLK, i < nbn ? &tmQn : &tmQr, bar, (i < nbn ? i : i - nbn) * 64, it.head[t], it.q0[t], 0, 0);
  }
  struct Step {
    int row;
    __device__ __forceinline__ Step(const LatentPrefillTc& p, const Item& it, int key0) : row(p.cu_k[it.b] + key0) {}
  };
  __device__ __forceinline__ void load_k(unsigned char* dst, uint64_t* bar, const Item& it, const Step& s, int i) const {
    if (i < nbn) tma_load_5d(dst, &tmKn, bar, i * 64, it.hk, s.row, 0, 0);
    else tma_load_5d(dst, &tmKr, bar, (i - nbn) * 64, 0, s.row, 0, 0);
  }
  __device__ __forceinline__ void load_v(unsigned char* dst, uint64_t* bar, const Item& it, const Step& s, int i) const {
    tma_load_5d(dst, &tmV, bar, i * 64, it.hk, s.row, 0, 0);
  }
  __device__ __forceinline__ T* out(int row, int head, int c) const { return o + (int64_t)row * out_stride + (int64_t)head * dv + c; }

  struct Row {
    int lim;
    float ref0;
    Factor fac;
    __device__ __forceinline__ Row(const LatentPrefillTc& p, const Item& it, int t, int r)
        : lim(min(it.keys - 1, of_tile(it.pos, t) + r)), ref0(-INFINITY), fac(p.scale_log2e) {}
    __device__ __forceinline__ float finish(const LatentPrefillTc&, float, float l) const { return l > 0.f ? 1.f / l : 0.f; }
  };
};

// Launches of up to so many 128-row query tiles (about: the counts are on the device) take the kernel of zp_latent_prefill_tc_short.cu.
// Kernel times of the two, 16 and 32 heads of 128 + 64 (us, this file / short): 32 tiles 13 / 11; 176: 23 to 36 / 13 to 29; 352: 29 to
// 47 / 22 to 39; 448, equal portions 32 / 40, continued ones 67 / 58; 512: 48 to 76 / 57 to 75, 128-token portions 64 / 48; 560: 52 to
// 98 / 73 to 112; 1216: 122 to 178 / 187 to 236.  (Measured with one group of softmax warps a tile here; two are up to 3 % faster.)
constexpr int64_t LATENT_SHORT = 512;
// Portions of up to one tile leave the second tile of every item empty, which costs the more the longer the work on the first lasts: with
// a context of four times the portions such launches go there too, whatever their number.  32 portions of 128, 100, 64, 32 tokens,
// 32 heads (us, this file / short): no context 59 / 74, 61 / 76, 59 / 70, 61 / 64; after 256 keys 105 / 107, 106 / 109, 107 / 102, 107 / 96; after
// 512 145 / 139, 146 / 143, 147 / 135, 148 / 131; after 2000 (128, 100, 64) 381 / 340, 383 / 338, 383 / 332.
static bool latent_takes_short(int H, int B, int max_seqlen_q, int total_q, int total_k) {
  return (int64_t)H * (total_q / 128 + B) <= LATENT_SHORT || (max_seqlen_q <= 128 && total_k >= (int64_t)5 * total_q);
}
int latent_prefill_tc_short(const void* q, int64_t q_stride, const void* kv, const void* latent, const int32_t* cu_seqlens_q, const int32_t* cu_seqlens_k,
                            void* out, int64_t out_stride, int B, int max_seqlen_q, int total_q, int total_k, int H, int dim, int rot, int vdim,
                            int kv_rank, int KP, float scale, cudaStream_t st);

}  // namespace zp

extern "C" int zp_latent_prefill_supported(int dim, int rot, int vdim, int kv_rank, int KP, int dtype) {
  const int nbq = (dim + 63) / 64 + (rot + 63) / 64;
  return dtype == ZP_DTYPE_BF16 && dim > 0 && vdim > 0 && vdim <= 128 && nbq <= 4 && dim % 8 == 0 && rot % 8 == 0 && vdim % 8 == 0 &&
         kv_rank % 8 == 0 && KP % 8 == 0;
}

extern "C" int zp_latent_prefill(const void* q, int64_t q_stride, const void* kv, const void* latent, const int32_t* cu_seqlens_q,
                                 const int32_t* cu_seqlens_k, void* out, int64_t out_stride, int B, int max_seqlen_q, int total_q,
                                 int total_k, int H, int dim, int rot, int vdim, int kv_rank, int KP, float scale, int dtype,
                                 void* stream) {
  using namespace zp;
  using namespace zp::tc;
  if (B == 0 || max_seqlen_q == 0) return ZP_OK;
  ZP_REQUIRE(q && kv && (latent || rot == 0) && cu_seqlens_q && cu_seqlens_k && out, "zp_latent_prefill: null pointer");
  ZP_REQUIRE(H > 0 && H <= 65535 && B <= 65535 && total_q > 0 && total_k > 0 && KP >= kv_rank + rot, "zp_latent_prefill: bad sizes");
  if (!zp_latent_prefill_supported(dim, rot, vdim, kv_rank, KP, dtype) || q_stride % 8 || out_stride % 8 ||
      ((uintptr_t)q | (uintptr_t)kv | (uintptr_t)latent | (uintptr_t)out) % 16) {
    set_error("zp_latent_prefill: needs bf16, head sizes that are multiples of 8 (values at most 128) and 16-byte aligned rows");
    return ZP_ERR_UNSUPPORTED;
  }
  // (the other kernel masks products before it scales them: factors above zero only)
  if (scale > 0.f && latent_takes_short(H, B, max_seqlen_q, total_q, total_k))
    return latent_prefill_tc_short(q, q_stride, kv, latent, cu_seqlens_q, cu_seqlens_k, out, out_stride, B, max_seqlen_q, total_q, total_k, H, dim,
                                   rot, vdim, kv_rank, KP, scale, (cudaStream_t)stream);
  LatentPrefillTc p;
  p.cu_q = cu_seqlens_q; p.cu_k = cu_seqlens_k; p.o = (__nv_bfloat16*)out; p.dv = vdim;
  p.nbn = (dim + 63) / 64;
  p.rings = rings_of(p.nbn + (rot + 63) / 64, (vdim + 63) / 64);
  p.mode = PAIR_ROWS;      // (every head has keys of its own)
  const dim3 grid = grid_of(p.mode, H, B, max_seqlen_q, p.levels);
  p.out_stride = out_stride; p.scale_log2e = scale * LOG2E;
  p.error_word = device_error_word();
  if (!p.error_word) { set_error("zp_latent_prefill: no device error word"); return ZP_ERR_CUDA; }
  const auto fmt = UmmaFmt<__nv_bfloat16>::tm;
  const __nv_bfloat16* qb = (const __nv_bfloat16*)q;
  const __nv_bfloat16* kb = (const __nv_bfloat16*)kv;
  const uint64_t kv_stride = (uint64_t)H * (dim + vdim), hd = dim + rot, qs = q_stride;
  const uint64_t uq = total_q, uk = total_k, uh = H;
  const uint32_t box[5] = {64, 1, 128, 1, 1};
  const uint64_t sq[4] = {hd, qs, qs * uq, qs * uq}, sk[4] = {(uint64_t)dim, kv_stride, kv_stride * uk, kv_stride * uk},
                 sv[4] = {(uint64_t)vdim, kv_stride, kv_stride * uk, kv_stride * uk},
                 sl[4] = {(uint64_t)KP, (uint64_t)KP, (uint64_t)KP * uk, (uint64_t)KP * uk};
  const uint64_t dqn[5] = {(uint64_t)dim, uh, uq, 1, 1}, dqr[5] = {(uint64_t)rot, uh, uq, 1, 1}, dkn[5] = {(uint64_t)dim, uh, uk, 1, 1},
                 dkr[5] = {(uint64_t)rot, 1, uk, 1, 1}, dv[5] = {(uint64_t)vdim, uh, uk, 1, 1};
  if (int rc = make_tensor_map_5d(&p.tmQn, fmt, qb, dqn, sq, box, 2)) return rc;
  if (int rc = make_tensor_map_5d(&p.tmKn, fmt, kb, dkn, sk, box, 2)) return rc;
  if (int rc = make_tensor_map_5d(&p.tmV, fmt, kb + (int64_t)H * dim, dv, sv, box, 2)) return rc;
  p.tmQr = p.tmQn;
  p.tmKr = p.tmKn;
  if (rot) {
    if (int rc = make_tensor_map_5d(&p.tmQr, fmt, qb + dim, dqr, sq, box, 2)) return rc;
    if (int rc = make_tensor_map_5d(&p.tmKr, fmt, (const __nv_bfloat16*)latent + kv_rank, dkr, sl, box, 2)) return rc;
  }
  return launch_attn(p, grid, (cudaStream_t)stream, "zp_latent_prefill");
}

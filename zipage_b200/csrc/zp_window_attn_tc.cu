// Prefill attention with masks (sliding window, chunks, kept keys), soft cap, distance biases, sink and output gate on tcgen05
// tensor cores: bf16, key and value sizes up to 128, paged caches (page size a multiple of 64).
//
// The pipeline is the one of zp_attn_tc.cuh, with the weights as bf16 hi + lo, over the visible key tiles (those of the
// kept keys first).  A soft cap bounds every score, so its reference is fixed (the cap, or 0; see zp_window_attn_mma.cu).
// A work item is two heads of one key/value head over the same 128 queries, or, where a key/value head has an odd number
// of heads, two neighbouring query tiles of one head.
//
// A key tile is two 64-key boxes per 64 entries, so its halves may lie in different pages; head sizes that are no
// multiples of 64 are filled with zeros by TMA.  The capped softmax takes two exponentials and a reciprocal per score; four reciprocals share
// one instruction, 1/a = bcd / (abcd).  It is bound by its instructions, not by the special-function unit: with a quarter of the exponentials as
// polynomials the call took 382 us instead of 367.
//
// A tile of its own per block, all softmax warps on it, left the tensor cores idle during each of its softmax turns.  Four portions of
// 500 to 3000 tokens, 32 heads on 8, window 1024, cap 30: 302 us (344 so).  Uniform portions, no window: 4 x 2000 tokens 236 us (320),
// 4 x 1000 85 (112); cap 30 and window 512: 86 (107).  Since then weights are handed over 32 keys at a time and split in fp32 (capped), and uncapped
// windows have two groups of softmax warps: the first of these 309 -> 286 us in one profiler, without cap 7 us less than with one group.
#include <algorithm>

#include "zp_attn_tc.cuh"
#include "zp_window_tc.cuh"

namespace zp {

using namespace attn;

template <bool CAPPED_, bool BIASED_>   // (not both)
struct WindowTc {
  using T = __nv_bfloat16;
  static constexpr bool SPLIT = true, MASKED = true, CAPPED = CAPPED_, BIASED = BIASED_, GATED = true;
  static constexpr int GROUPS = BIASED_ ? 1 : 2;
  static constexpr float LAZY = 40.f;
  CUtensorMap tmQ, tmK, tmV;
  WinArgs a;
  int* error_word;
  Rings rings;
  int levels, dv, mode;

  __device__ __forceinline__ void prefetch() const {
    prefetch_tensormap(&tmQ);
    prefetch_tensormap(&tmK);
    prefetch_tensormap(&tmV);
  }
  __device__ __forceinline__ bool item(dim3 id, Item& it) const {
    const WinSeq sq = win_seq(a, id.y);
    const int first = (levels - 1 - (int)id.z) * level_rows(mode);
    if (first >= sq.count) return false;
    it.b = id.y;
    it.keys = sq.ctx;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int qi = item_row(mode, first, t);
      it.head[t] = item_head(mode, id.x, t);
      it.q0[t] = sq.row0 + qi;
      it.rows[t] = item_rows(mode, sq.count - qi, t);
      it.pos[t] = sq.pos0 + qi;
      const WinTiles w = win_tiles(a, it.pos[0], it.pos[t] + it.rows[t] - 1, 128);
      it.n[t] = it.rows[t] > 0 ? w.n : 0;
      if (t == 0) { it.kept = w.kept; it.t0 = w.t0; }
    }
    it.hk = it.head[0] / (a.Hq / a.Hkv);
    return true;
  }
  __device__ __forceinline__ void load_q(unsigned char* dst, uint64_t* bar, const Item& it, int t) const {
    for (int i = 0; i < rings.nbq; ++i) tma_load_5d(dst + i * BLK, &tmQ, bar, i * 64, it.head[t], it.q0[t], 0, 0);
  }
  struct Step {
    int row[2], page[2];      // of the two halves
    __device__ __forceinline__ Step(const WindowTc& p, const Item& it, int key0) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        row[u] = (key0 + 64 * u) % p.a.BS;
        page[u] = win_page(p.a, it.b, key0 + 64 * u);
      }
    }
  };
  __device__ __forceinline__ void load_kv(unsigned char* dst, const CUtensorMap* tm, uint64_t* bar, const Item& it, const Step& s, int i) const {
#pragma unroll
    for (int u = 0; u < 2; ++u) tma_load_5d(dst + u * (BLK / 2), tm, bar, i * 64, it.hk, s.row[u], s.page[u], 0);
  }
  __device__ __forceinline__ void load_k(unsigned char* dst, uint64_t* bar, const Item& it, const Step& s, int i) const { load_kv(dst, &tmK, bar, it, s, i); }
  __device__ __forceinline__ void load_v(unsigned char* dst, uint64_t* bar, const Item& it, const Step& s, int i) const { load_kv(dst, &tmV, bar, it, s, i); }
  __device__ __forceinline__ T* out(int row, int head, int c) const {
    return reinterpret_cast<T*>(a.out) + (int64_t)row * a.out_stride + (int64_t)head * a.DV + c;
  }

  struct Row {
    int lim, lo, keep, row, head;
    bool real;
    float ref0, y, m2c, off, slope;
    Factor fac;
    __device__ __forceinline__ Row(const WindowTc& p, const Item& it, int t, int r)
        : lim(of_tile(it.pos, t) + r), lo(win_first(p.a, lim)), keep(p.a.keep), row(of_tile(it.q0, t) + r), head(of_tile(it.head, t)),
          real(r < of_tile(it.rows, t)), ref0(-INFINITY), fac(p.a.scale * LOG2E) {
      if constexpr (CAPPED) {
        y = 2.f * LOG2E * p.a.scale / p.a.softcap;
        m2c = -2.f * p.a.softcap * LOG2E;
        off = -2.f * m2c <= 200.f ? 0.f : -0.5f * m2c;      // cap minus reference
        ref0 = -0.5f * m2c - off;
      }
      if constexpr (BIASED) slope = win_slope2(p.a, head);
    }
    __device__ __forceinline__ void transform(uint32_t (&s)[32], int key0) const {
      const float at = slope * (float)(key0 - lim);      // bias of the first column (lim is the row's position)
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        float2 x = make_float2(fmaf(slope, (float)i, at), fmaf(slope, (float)(i + 1), at));
        ffma2(x, make_float2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), make_float2(fac.mag, fac.mag));
        s[i] = __float_as_uint(x.x);
        s[i + 1] = __float_as_uint(x.y);
      }
    }
    __device__ __forceinline__ void weights4(const uint32_t* s, float (&w)[4]) const { zp::weights4(s, y, m2c, off, w); }
    __device__ __forceinline__ float finish(const WindowTc& p, float ref, float l) const {
      if (!real) return 0.f;
      if (p.a.sink) l += ex2_approx(win_sink2(p.a, head) - ref);
      return l > 0.f ? win_head_factor<T>(p.a, row, head) / l : 0.f;
    }
    __device__ __forceinline__ void entries(const WindowTc& p, int c, float (&v)[32]) const {
      if (p.a.gate_mode != WIN_GATE_ENTRY || !real) return;
      const T* gate = reinterpret_cast<const T*>(p.a.gate) + (int64_t)row * p.a.gate_stride + (int64_t)head * p.a.DV + c;
#pragma unroll
      for (int i = 0; i < 32; i += 8) {
        if (c + i >= p.a.DV) break;
        const int4 raw = ld16(gate + i);
        const T* ge = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int u = 0; u < 8; ++u) v[i + u] *= win_sigmoid(__bfloat162float(ge[u]));
      }
    }
  };
};

// whether the kernel can run this call (total_q: rows of q)
bool window_tc_supports(const WinArgs& a, int total_q, int dtype) {
  return dtype == ZP_DTYPE_BF16 && a.KP <= 128 && a.VP <= 128 && a.D % 8 == 0 && a.DV % 8 == 0 && total_q > 0 &&
         a.softcap * 1.4426950408889634f <= 100.f && !(a.slopes && a.softcap > 0.f) && a.q_stride % 8 == 0 && a.out_stride % 8 == 0 &&
         (a.gate_mode != WIN_GATE_ENTRY || (a.gate_stride % 8 == 0 && (uintptr_t)a.gate % 16 == 0)) &&
         ((uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.out) % 16 == 0;
}

template <class P>
static int launch_window_tc(const WinArgs& a, int max_q, int total_q, cudaStream_t st) {
  P p;
  p.a = a;
  p.error_word = device_error_word();
  if (!p.error_word) { set_error("zp_window_attention(tcgen05): no device error word"); return ZP_ERR_CUDA; }
  const auto fmt = UmmaFmt<__nv_bfloat16>::tm;
  {
    const uint64_t dims[5] = {(uint64_t)a.D, (uint64_t)a.Hq, (uint64_t)total_q, 1, 1};
    const uint64_t strides[4] = {(uint64_t)a.D, (uint64_t)a.q_stride, (uint64_t)a.q_stride, (uint64_t)a.q_stride};
    const uint32_t box[5] = {64, 1, 128, 1, 1};
    if (int rc = make_tensor_map_5d(&p.tmQ, fmt, a.q, dims, strides, box, 2)) return rc;
  }
  const uint32_t box[5] = {64, 1, 64, 1, 1};
  for (int kv = 0; kv < 2; ++kv) {
    const uint64_t w = kv ? a.VP : a.KP, row = (uint64_t)a.Hkv * w, page = (uint64_t)a.BS * row;
    const uint64_t dims[5] = {w, (uint64_t)a.Hkv, (uint64_t)a.BS, (uint64_t)a.n_pages, 1};
    const uint64_t strides[4] = {w, row, page, page};
    if (int rc = make_tensor_map_5d(kv ? &p.tmV : &p.tmK, fmt, kv ? a.v : a.k, dims, strides, box, 2)) return rc;
  }
  p.rings = rings_of((a.D + 63) / 64, (a.DV + 63) / 64);
  p.dv = a.DV;
  p.mode = pick_pair(a.Hq / a.Hkv);
  const dim3 grid = grid_of(p.mode, a.Hq, a.B, max_q, p.levels);
  return launch_attn(p, grid, st, "zp_window_attention(tcgen05)");
}

// Launches of few 128-row query tiles take the kernel of zp_window_attn_tc_short.cu (single tiles, whose waves are finer and whose code is
// shorter to fetch).  Times of this file's kernel over that one's, heads of 128, portions of 96 to 2560 tokens, 32 heads on 8 unless noted; the
// lines lie where no column is above 1 by more than a few percent.  (Measured before this file's kernel became 3 to 7 % faster: a call
// just below a line may now take the slower kernel by as much.)
//   tiles        no context, no cap   cap   | window 512 or 1024, context 2000: no cap   cap   | no window, context 2000: no cap   cap
//   320 .. 416   0.86 .. 1.00   0.91 .. 1.03 | 1.05 .. 1.14   1.12 .. 1.20                     | 0.95 .. 1.18   1.13 .. 1.26
//   448 .. 576   0.70 .. 0.76   0.72 .. 0.82 | 0.83 .. 0.90   0.90 .. 0.97                     | 0.82 .. 0.96   0.90 .. 0.99
//   608 .. 736   0.75 .. 0.84   0.76 .. 0.96 | 0.91 .. 0.98   1.02 .. 1.06                     | 0.91 .. 1.01   1.02 .. 1.15
//   768 ..       0.60 .. 0.83   0.63 .. 0.82 | 0.80 .. 0.94   0.84 .. 0.99                     | 0.78 .. 0.92   0.84 .. 1.01 (one 1.09)
// (Caps: two waves of pairs last as long as three to four of single tiles, so 608 to 736 tiles, three waves for five, lose.)  With an odd
// number of heads per key/value head a pair is two row blocks of one head: half empty for portions of one tile (1.14 to 1.35 with a context
// of 500 to 2000 keys), and under a window or behind a context each of its tiles also walks keys that only the other one sees (16 heads on
// 16, 12 portions of 30 to 1500 tokens after 1000, window 512: 1.07 to 1.11; 48 of 10 to 200: 1.24 to 1.28).  Without either it
// is 0.67 to 1.00.
constexpr int64_t WINDOW_SHORT = 704;      // in heads x (rows / 128 + portions), at most twice the number of tiles
constexpr int64_t WINDOW_TILES = 432, WINDOW_TILES_CAP = 768;
int window_prefill_tc_short(const WinArgs& a, int max_q, int total_q, cudaStream_t st);

static bool window_takes_short(const WinArgs& a, int max_q, int total_q, bool forced) {
  if ((int64_t)a.Hq * (total_q / 128 + a.B) <= WINDOW_SHORT) return true;
  if (forced) return false;
  const int64_t keys = (int64_t)a.NBmax * a.BS;      // that a sequence's table has room for
  if (a.Hq / a.Hkv % 2) return a.window > 0 || a.chunk > 0 || 2 * keys >= (int64_t)3 * max_q;
  // tiles: half a tile more per portion than its rows fill, at most what the longest portion has (the counts are on the device)
  const int64_t tiles = a.Hq * std::min((int64_t)a.B * ((max_q + 127) / 128), std::max((int64_t)a.B, (int64_t)total_q / 128 + (a.B + 1) / 2));
  if (tiles < WINDOW_TILES) return true;
  const int64_t span = std::min({keys, a.window > 0 ? (int64_t)a.window : keys, a.chunk > 0 ? (int64_t)a.chunk : keys});
  const bool far = span < keys ? span >= 512 : span > 1024;      // a row sees so many keys
  return a.softcap > 0.f && far && tiles < WINDOW_TILES_CAP;
}

// forced: the caller asked for tcgen05 (lines that depend on more than the number of tiles are for the others)
int window_prefill_tc(const WinArgs& a, int max_q, int total_q, bool forced, cudaStream_t st) {
  // (the other kernel masks products before it scales them: factors above zero only)
  if ((a.scale > 0.f || a.softcap > 0.f) && window_takes_short(a, max_q, total_q, forced)) return window_prefill_tc_short(a, max_q, total_q, st);
  if (a.softcap > 0.f) return launch_window_tc<WindowTc<true, false>>(a, max_q, total_q, st);
  if (a.slopes) return launch_window_tc<WindowTc<false, true>>(a, max_q, total_q, st);
  return launch_window_tc<WindowTc<false, false>>(a, max_q, total_q, st);
}

}  // namespace zp

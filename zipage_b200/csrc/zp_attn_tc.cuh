// Softmax attention of many queries on tcgen05 tensor cores: the pipeline that the kernels over whole prompts, windows and
// expanded latents share.  A kernel brings a parameter struct P that says which tiles there are, where their
// operands lie and which keys a row sees; everything else is here.
//
// A work item is two tiles of 128 query rows that meet the same 128-key tiles: two heads of one key/value head, or
// neighbouring rows of one head.  Each key tile is fetched once for both, and while the softmax works on one
// tile's scores the tensor cores work on the other's:
//   S_t = Q_t K^T                [128 queries, 128 keys] fp32 in TMEM
//   p = exp2(s - m)              fp32; as T, or as two bf16 numbers (hi + lo), over S_t's own columns
//   O_t += p V                   [128 queries, up to 128 entries] fp32 in TMEM
// and at the end O / row sum.  m is one reference per row: the maximum of the first tile, moved (and O with it) only
// when a score exceeds it by more than P::LAZY powers of two, which floats of either size carry without loss; a kernel
// whose scores are bounded has a fixed one.
//
// What bounds it: per 128 x 128 scores the two products take 1024 clocks of the tensor pipe (1536 with hi + lo) and the
// exponentials 1024 of the special-function unit, so neither may wait for the other; two tiles in flight hide the
// softmax's latency, and as a thread owns a whole row no maximum or sum ever crosses threads.
//
// Roles (three warpgroups, one block per SM): warp 0 = TMA producer and TMEM owner, warp 1 = MMA issuer, warps 4-7 and 8-11 =
// softmax of tile 0 and 1, which take over registers of the first group (a row's 128 scores stay in them).  The MMAs of one issuing thread run in order, so S_t of the next key tile may be issued
// right behind the product that reads p from the same columns.  Shared memory: both query tiles, a ring of 16 KB key
// blocks (128 keys x 64 entries), a ring of value tiles.
//
// Blocks stay: each takes over the grid's tiles that have not started yet (cluster launch control), so that the next
// item's queries and keys arrive during the last softmax and the output of the item before.  The grid's order is
// the order of the work: levels of equal length, the longest first.
// Every wait is bounded; after one that runs out the block raises the device error word and leaves.
#pragma once
#include "zp_tc.cuh"

namespace zp {
namespace attn {

using namespace tc;

constexpr int THREADS = 384;
constexpr int REGS_FEED = 72, REGS_SOFTMAX = 216;      // of 168 a thread at launch: 72 + 2 x 216 = 3 x 168
constexpr int BLK = 16384;               // 128 rows x 64 elements x 2 bytes
constexpr int MAXRING = 12;
constexpr uint32_t O_COL = 256;          // TMEM columns: S_0 | S_1 | O_0 | O_1, 128 each
constexpr int SLACK = 128;               // alignment padding that the launch provides for
constexpr float LOG2E = 1.4426950408889634f;

struct __align__(16) Shared {
  uint4 work[2];                         // answers of cluster launch control
  uint64_t wfull[2], wempty[2], qfull, qempty, kfull[MAXRING], kempty[MAXRING], vfull[MAXRING], vempty[MAXRING], sfull[2], pfull[2], pvdone[2];
  uint32_t tmem_base;
  int abort_flag;
};

// Two tiles of one sequence.
struct Item {
  int b, head[2], hk;                    // sequence, query head of each tile, key/value head
  int q0[2], rows[2], pos[2];            // first row of q (absolute), rows, position of the first row
  int keys;                              // keys of the sequence: rows past them are not read
  int n[2];                              // key tiles 0 .. n - 1 of each
  int kept, t0;                          // key tile j is number j < kept ? j : t0 + j - kept
  __device__ __forceinline__ int most() const { return max(n[0], n[1]); }
  __device__ __forceinline__ int last(int j) const { return j < n[1] ? 1 : 0; }      // the tiles that take part in step j: the later one, ...
  __device__ __forceinline__ int first(int j) const { return j < n[0] ? 0 : 1; }     // ... and the earlier one
  __device__ __forceinline__ int key0(int j) const { return (j < kept ? j : t0 + j - kept) * 128; }
};
template <typename V> __device__ __forceinline__ V of_tile(const V (&a)[2], int t) { return t ? a[1] : a[0]; }      // (an index would put a in memory)
struct Rings { int nbq, nbv, nk, nv; };  // 64-entry blocks of a query (key) row and of a value row; key blocks and value tiles in the rings

// ---- cluster launch control ---------------------------------------------------------------------
__device__ __forceinline__ void ask_work(uint4* answer, uint64_t* bar) {
  mbar_arrive_expect_tx(bar, 16);
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(smem_u32(answer)),
               "r"(smem_u32(bar))
               : "memory");
}
// whether a block of the grid was taken over, and which
__device__ __forceinline__ bool read_work(const uint4* answer, dim3& id) {
  uint32_t ok, x = 0, y = 0, z = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 a;\n\t"
      "ld.shared.b128 a, [%4];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, a;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, %2, %3, _}, a;\n\t"
      "fence.proxy.async.shared::cta;\n\t}"
      : "=r"(ok), "+r"(x), "+r"(y), "+r"(z)
      : "r"(smem_u32(answer))
      : "memory");
  id = dim3(x, y, z);
  return ok != 0;
}

// ---- operands --------------------------------------------------------------------------------------
// MN-major tile, 128-byte swizzle: 64 contiguous elements per K row, 8-row groups 1024 bytes apart along K, the next 64
// elements along MN a block away
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr) {
  const uint32_t lo = ((addr >> 4) & 0x3FFFu) | ((uint32_t)(BLK >> 4) << 16);
  const uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);
  return (static_cast<uint64_t>(hi) << 32) | lo;
}
// A operand from TMEM (one row per lane, two 16-bit elements per column)
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d), "r"(a), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
// the same answer in all lanes of the warp
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* error_word, int where) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, error_word, where));
}

// What P has to bring:
//   T                            element type;  SPLIT: weights as hi + lo (T = bf16);  MASKED: rows have a first visible key too
//   LAZY                         powers of two by which a score may exceed its row's reference;  CAPPED: the reference is fixed
//   rings, error_word            members
//   item(id, it)                 the work of block `id`; false: none
//   load_q(dst, bar, it, t), load_k(dst, bar, it, key0, i), load_v(dst, bar, it, key0, i): TMA loads of one block each
//   Row(p, it, t, r)             one query row, with lim (last visible key) and, where MASKED, lo and keep (keys j < lo are not seen
//                                unless j < keep), ref0 (first reference; -inf unless CAPPED), and
//     scale()                    what a raw product is multiplied by to become the exponent of 2, or
//     transform(s, key0)         (P::BIASED) raw products of 32 keys to exponents of 2, or
//     weights4(s, w)             (CAPPED) four raw products to four weights
//     finish(p, ref, l)          factor of the row's sums (1 / l, gates)
//     entries(p, c, v)           (P::GATED) factors of 32 entries
//   out(row, head, c), dv        address of entry c of a row, entries of a head
template <class P>
__global__ void __launch_bounds__(THREADS, 1) attn_tc_kernel(const __grid_constant__ P p) {
  using T = typename P::T;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* qbuf = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  if (qbuf - smem_raw > SLACK) {         // (no room for more padding)
    if (threadIdx.x == 0) atomicCAS(p.error_word, 0, 820);
    return;
  }
  const Rings g = p.rings;
  unsigned char* kring = qbuf + 2 * g.nbq * BLK;
  unsigned char* vring = kring + g.nk * BLK;
  Shared& sh = *reinterpret_cast<Shared*>(vring + g.nv * g.nbv * BLK);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh.wfull[i], 1); mbar_init(&sh.wempty[i], 10);
      mbar_init(&sh.sfull[i], 1); mbar_init(&sh.pfull[i], 4); mbar_init(&sh.pvdone[i], 1);
    }
    mbar_init(&sh.qfull, 1); mbar_init(&sh.qempty, 1);
    for (int i = 0; i < g.nk; ++i) { mbar_init(&sh.kfull[i], 1); mbar_init(&sh.kempty[i], 1); }
    for (int i = 0; i < g.nv; ++i) { mbar_init(&sh.vfull[i], 1); mbar_init(&sh.vempty[i], 1); }
    sh.abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(&sh.tmem_base, 512);
    tmem_relinquish();
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = sh.tmem_base;
  volatile int* abortp = &sh.abort_flag;
  dim3 id(blockIdx.x, blockIdx.y, blockIdx.z);
  Item it;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_FEED));
    if (warp == 0 && elect_one()) {
      uint32_t kslot = 0, kround = 0, vslot = 0, vround = 0, nq = 0;
      bool ok = true;
      for (uint32_t w = 0; ok; ++w) {
        ok = mbar_wait(&sh.wempty[w & 1], ((w >> 1) & 1) ^ 1, abortp, p.error_word, 821);
        if (!ok) break;
        ask_work(&sh.work[w & 1], &sh.wfull[w & 1]);
        if (p.item(id, it) && it.most() > 0) {
          ok = mbar_wait<true>(&sh.qempty, (nq & 1) ^ 1, abortp, p.error_word, 822);
          if (!ok) break;
          mbar_arrive_expect_tx(&sh.qfull, (uint32_t)(((it.n[0] > 0) + (it.n[1] > 0)) * g.nbq * BLK));
#pragma unroll
          for (int t = 0; t < 2; ++t)
            if (it.n[t] > 0) p.load_q(qbuf + t * g.nbq * BLK, &sh.qfull, it, t);
          ++nq;
          for (int j = 0; ok && j < it.most(); ++j) {
            const int key0 = it.key0(j);
            for (int i = 0; i < g.nbq; ++i) {
              if (!mbar_wait<true>(&sh.kempty[kslot], (kround & 1) ^ 1, abortp, p.error_word, 823)) { ok = false; break; }
              mbar_arrive_expect_tx(&sh.kfull[kslot], BLK);
              p.load_k(kring + kslot * BLK, &sh.kfull[kslot], it, key0, i);
              if (++kslot == (uint32_t)g.nk) { kslot = 0; ++kround; }
            }
            if (!ok || !mbar_wait<true>(&sh.vempty[vslot], (vround & 1) ^ 1, abortp, p.error_word, 824)) { ok = false; break; }
            mbar_arrive_expect_tx(&sh.vfull[vslot], (uint32_t)(g.nbv * BLK));
            for (int i = 0; i < g.nbv; ++i) p.load_v(vring + (vslot * g.nbv + i) * BLK, &sh.vfull[vslot], it, key0, i);
            if (++vslot == (uint32_t)g.nv) { vslot = 0; ++vround; }
          }
          if (!ok) break;
        }
        // (also after a refusal: the answer has to arrive before the block may end)
        ok = mbar_wait(&sh.wfull[w & 1], (w >> 1) & 1, abortp, p.error_word, 825) && read_work(&sh.work[w & 1], id);
        mbar_arrive(&sh.wempty[w & 1]);
      }
    }
    if (warp == 1 && elect_one()) {
      constexpr uint32_t ID_S = idesc_f16(UmmaFmt<T>::fmt, 128, 128);
      const uint32_t id_o = idesc_f16(UmmaFmt<T>::fmt, 128, 64 * g.nbv) | (1u << 16);      // V is MN-major
      const uint32_t q_addr = smem_u32(qbuf), k_addr = smem_u32(kring), v_addr = smem_u32(vring);
      uint32_t cnt[2] = {0, 0}, kslot0 = 0, kround0 = 0, vslot = 0, vround = 0, nq = 0;      // (key blocks of step 0 of an item, value tile)
      bool ok = true;
      for (uint32_t w = 0; ok; ++w) {
        if (p.item(id, it) && it.most() > 0) {
          const int most = it.most();
          ok = mbar_wait(&sh.qfull, nq & 1, abortp, p.error_word, 826);
          ++nq;
          uint32_t ks_[2] = {kslot0, kslot0}, kr_[2] = {kround0, kround0};      // where each tile is in the key ring
          auto issue_s = [&](int t, int j) -> bool {
            const bool release = t == it.last(j);
            uint32_t s = ks_[t], r = kr_[t];
            for (int i = 0; i < g.nbq; ++i) {
              if (!mbar_wait(&sh.kfull[s], r & 1, abortp, p.error_word, 827)) return false;
              fence_after_sync();
              const uint64_t ad = smem_desc_sw128(q_addr + (t * g.nbq + i) * BLK), bd = smem_desc_sw128(k_addr + s * BLK);
#pragma unroll
              for (int k = 0; k < 4; ++k) umma_f16(tmem + t * 128, ad + 2u * k, bd + 2u * k, ID_S, (i | k) ? 1u : 0u);
              if (release) umma_commit(&sh.kempty[s]);
              if (++s == (uint32_t)g.nk) { s = 0; ++r; }
            }
            ks_[t] = s; kr_[t] = r;
            if (release) { kslot0 = s; kround0 = r; }
            umma_commit(&sh.sfull[t]);
            if (j == most - 1 && release) umma_commit(&sh.qempty);
            return true;
          };
#pragma unroll
          for (int t = 0; t < 2; ++t)
            if (ok && it.n[t] > 0) ok = issue_s(t, 0);
#pragma unroll 1
          for (int j = 0; ok && j < most; ++j) {
#pragma unroll
            for (int t = 0; t < 2; ++t) {
              if (!ok || j >= it.n[t]) continue;
              if (t == it.first(j)) ok = mbar_wait(&sh.vfull[vslot], vround & 1, abortp, p.error_word, 828);
              if (!ok || !mbar_wait(&sh.pfull[t], cnt[t] & 1, abortp, p.error_word, 829)) { ok = false; continue; }
              fence_after_sync();
              const uint32_t v0 = v_addr + vslot * g.nbv * BLK, pt = tmem + t * 128, ot = tmem + O_COL + t * 128;
#pragma unroll
              for (int ks = 0; ks < 8; ++ks) {      // 16 keys a step: 8 columns of p
                const uint64_t bd = desc_mn(v0 + ks * 2048);
                umma_ts(ot, pt + ks * 8, bd, id_o, (j | ks) ? 1u : 0u);
                if (P::SPLIT) umma_ts(ot, pt + 64 + ks * 8, bd, id_o, 1u);
              }
              if (t == it.last(j)) umma_commit(&sh.vempty[vslot]);
              umma_commit(&sh.pvdone[t]);
              ++cnt[t];
              if (j + 1 < it.n[t]) ok = issue_s(t, j + 1);
            }
            if (++vslot == (uint32_t)g.nv) { vslot = 0; ++vround; }
          }
          if (!ok) break;
        }
        ok = mbar_wait(&sh.wfull[w & 1], (w >> 1) & 1, abortp, p.error_word, 830) && read_work(&sh.work[w & 1], id);
        mbar_arrive(&sh.wempty[w & 1]);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_SOFTMAX));
    const int t = (warp - 4) >> 2, quad = warp & 3, r = quad * 32 + lane;      // tile, TMEM lane quadrant, row of the tile
    const uint32_t lanes = tmem + (static_cast<uint32_t>(quad * 32) << 16), st = lanes + t * 128, ot = lanes + O_COL + t * 128;
    uint32_t cnt = 0, vslot = 0, vround = 0;
    bool ok = true;
    for (uint32_t w = 0; ok; ++w) {
      if (p.item(id, it)) {
        const int n = of_tile(it.n, t), most = it.most();
        const typename P::Row row(p, it, t, r);
        float2 l2 = make_float2(0.f, 0.f);
        float ref = row.ref0;
        for (int j = 0; ok && j < n; ++j) {
          const int key0 = it.key0(j);
          ok = warp_wait(&sh.sfull[t], cnt & 1, abortp, p.error_word, 831);
          if (!ok) break;
          fence_after_sync();
          uint32_t s[4][32];
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld32_issue(st + c * 32, s[c]);
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld32_wait(s[c]);
          bool whole = key0 + 127 <= row.lim;
          if constexpr (P::MASKED) whole = whole && (key0 >= row.lo || key0 + 128 <= row.keep);
          whole = __all_sync(0xffffffffu, whole);
          if constexpr (P::BIASED) {
#pragma unroll
            for (int c = 0; c < 4; ++c) row.transform(s[c], key0 + c * 32);
          }
          if (!whole && !P::CAPPED) {
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const int key = key0 + c * 32 + i;
                bool seen = key <= row.lim;
                if constexpr (P::MASKED) seen = seen && (key >= row.lo || key < row.keep);
                if (!seen) s[c][i] = 0xff800000u;      // -inf
              }
          }
          if constexpr (!P::CAPPED) {
            float mx[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              mx[c] = fmaxf(__uint_as_float(s[c][0]), __uint_as_float(s[c][1]));
#pragma unroll
              for (int i = 2; i < 32; i += 2) mx[c] = fmax3(mx[c], __uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1]));
            }
            float m = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            if constexpr (!P::BIASED) m *= row.scale();
            const bool moves = m > ref + P::LAZY;
            if (__any_sync(0xffffffffu, moves)) {
              const float fac = moves ? ex2(ref - m) : 1.f;
              if (moves) ref = m;
              l2.x *= fac;
              l2.y *= fac;
              if (j > 0) {
                ok = warp_wait(&sh.pvdone[t], (cnt & 1) ^ 1, abortp, p.error_word, 832);
                if (!ok) break;
                fence_after_sync();
#pragma unroll 1
                for (int c = 0; c < 4 * g.nbv; ++c) {
                  uint32_t o[16];
                  tmem_ld16(ot + c * 16, o);
#pragma unroll
                  for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * fac);
                  tmem_st16(ot + c * 16, o);
                }
              }
            }
          }
          const float mref = ref == -INFINITY ? 0.f : ref;      // (no key seen so far: every weight is exp2(-inf))
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t hi[16], lo[16];
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              float wt[4];
              if constexpr (P::CAPPED) {
                row.weights4(&s[c][i], wt);
                if (!whole) {
#pragma unroll
                  for (int u = 0; u < 4; ++u) {
                    const int key = key0 + c * 32 + i + u;
                    bool seen = key <= row.lim;
                    if constexpr (P::MASKED) seen = seen && (key >= row.lo || key < row.keep);
                    if (!seen) wt[u] = 0.f;
                  }
                }
              } else {
                const float sc = P::BIASED ? 1.f : row.scale();
#pragma unroll
                for (int u = 0; u < 4; u += 2) {
                  float2 x = make_float2(-mref, -mref);
                  ffma2(x, make_float2(__uint_as_float(s[c][i + u]), __uint_as_float(s[c][i + u + 1])), make_float2(sc, sc));
                  wt[u] = ex2(x.x);
                  wt[u + 1] = ex2(x.y);
                }
              }
              l2 = fadd2(l2, fadd2(make_float2(wt[0], wt[1]), make_float2(wt[2], wt[3])));
#pragma unroll
              for (int u = 0; u < 4; u += 2) {
                const typename Pair<T>::V x = Pair<T>::pack(wt[u], wt[u + 1]);
                hi[(i + u) >> 1] = *reinterpret_cast<const uint32_t*>(&x);
                if constexpr (P::SPLIT) {
                  const float2 f = Pair<T>::unpack(x);
                  const typename Pair<T>::V z = Pair<T>::pack(wt[u] - f.x, wt[u + 1] - f.y);
                  lo[(i + u) >> 1] = *reinterpret_cast<const uint32_t*>(&z);
                }
              }
            }
            tmem_st16(st + c * 16, hi);
            if constexpr (P::SPLIT) tmem_st16(st + 64 + c * 16, lo);
          }
          // value rows past the sequence become zeros (0 times another sequence's values could be NaN)
          const int left = it.keys - key0;
          if (left < 128 && t == it.first(j)) {
            ok = warp_wait(&sh.vfull[vslot], vround & 1, abortp, p.error_word, 833);
            if (!ok) break;
            for (int i = r; i < (128 - left) * 8 * g.nbv; i += 128) {
              const int line = i >> 3, blk = line / (128 - left), key = left + line % (128 - left);
              *reinterpret_cast<int4*>(vring + (vslot * g.nbv + blk) * BLK + key * 128 + ((i & 7) << 4)) = make_int4(0, 0, 0, 0);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          }
          tmem_st_wait();
          fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.pfull[t]);
          ++cnt;
          if (++vslot == (uint32_t)g.nv) { vslot = 0; ++vround; }
        }
        if (!ok) break;
        for (int j = n; j < most; ++j)
          if (++vslot == (uint32_t)g.nv) { vslot = 0; ++vround; }
        // ---- output: four lanes share a row's 64 bytes ----
        if (n > 0) {
          ok = warp_wait(&sh.pvdone[t], (cnt & 1) ^ 1, abortp, p.error_word, 834);
          if (!ok) break;
          fence_after_sync();
        }
        const float inv = row.finish(p, ref, l2.x + l2.y);
        const int rows = of_tile(it.rows, t), q0 = of_tile(it.q0, t), head = of_tile(it.head, t), r4 = r & ~3, c8 = (lane & 3) * 8;
#pragma unroll 1
        for (int c = 0; c < 64 * g.nbv; c += 32) {
          uint32_t o[32];
          if (n > 0) {
            tmem_ld32_issue(ot + c, o);
            tmem_ld32_wait(o);
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = 0u;
          }
          float f[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) f[i] = inv * __uint_as_float(o[i]);
          if constexpr (P::GATED) row.entries(p, c, f);
          int4 v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint32_t x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const typename Pair<T>::V y = Pair<T>::pack(f[8 * i + 2 * u], f[8 * i + 2 * u + 1]);
              x[u] = *reinterpret_cast<const uint32_t*>(&y);
            }
            v[i] = make_int4((int)x[0], (int)x[1], (int)x[2], (int)x[3]);
          }
          transpose4(v, lane);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (r4 + i < rows && c + c8 < p.dv) st16(p.out(q0 + r4 + i, head, c + c8), v[i]);
        }
        fence_before_sync();      // (the next item's first product into O follows this warp's next arrival)
      }
      ok = warp_wait(&sh.wfull[w & 1], (w >> 1) & 1, abortp, p.error_word, 835) && read_work(&sh.work[w & 1], id);
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.wempty[w & 1]);
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

// ---- host ----------------------------------------------------------------------------------------------
// Rings for rows of nbq and nbv blocks: two value tiles (one where the queries take over half of the shared memory), the rest
// key blocks.  With two key blocks a row that is three key tiles and two value tiles; with three, 4 key blocks and two value tiles.
static inline Rings rings_of(int nbq, int nbv) {
  const int blocks = (232448 - SLACK - (int)sizeof(Shared)) / BLK - 2 * nbq;
  Rings g{nbq, nbv, 0, nbq > 3 ? 1 : 2};
  g.nk = blocks - g.nv * nbv;
  if (g.nk > MAXRING) g.nk = MAXRING;
  return g;
}

template <class P>
static int launch_attn(const P& p, dim3 grid, cudaStream_t st, const char* what) {
  const int smem = (2 * p.rings.nbq + p.rings.nk + p.rings.nv * p.rings.nbv) * BLK + (int)sizeof(Shared) + SLACK;
  cudaError_t e = cudaFuncSetAttribute(attn_tc_kernel<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) { set_error("%s: %s", what, cudaGetErrorString(e)); return ZP_ERR_CUDA; }
  attn_tc_kernel<P><<<grid, THREADS, smem, st>>>(p);
  return check_launch(what);
}

}  // namespace attn
}  // namespace zp

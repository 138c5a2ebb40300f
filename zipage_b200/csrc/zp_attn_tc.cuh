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
// What bounds it: the chain of a tile's step.  Per 128 x 128 scores the two products take 1024 clocks of the tensor pipe (1536 with hi +
// lo) and the exponentials 1024 of the special-function unit, but a step of two tiles takes 3500 to 4000: with one warp per 32
// rows 1040 clocks until the next scores are there (the rest of the second product, the first one, three hand-overs), 360 to load them,
// 310 for the maximum, 1870 for exponentials and weights (12 to 13 a pair of numbers; a third of all issue slots are used, a fifth of the
// warps' time goes into fetching instructions), 190 for the last hand-over.  On long prompts the clock falls from 1.83 to 1.6 GHz
// (power), so that instructions count as much as clocks.
//
// Softmax warps: P::GROUPS groups of four a tile.  One group: a thread owns a whole row and no maximum or sum ever crosses threads.
// Two groups split a row's keys and exchange its maximum through shared memory: half the loads, comparisons and exponentials follow
// one another, for half as many instructions again.  That is the better way for single tiles of few keys (see zp_prefill_tc.cu) and where a score costs more
// (calls with uncapped windows 334 -> 325 us, latents 476 -> 470; capped windows have no maximum to exchange and meet at an item's end alone), and the
// worse one for single tiles of many keys, pairs of tiles of long prompts (16384 tokens 2.29 -> 2.36 ms) and biased windows (385 -> 421).
//
// Roles (one block per SM): warp 0 = work, TMA loads and TMEM, warp 1 = products, from warp 4 on softmax, P::GROUPS groups of
// four warps a tile, which take over registers of the first group.  One thread issues the
// products of both tiles in turn, which keeps them half a step apart (with an issuer per tile they fell into step and
// overlapped less: 2.43 ms at 1 x 16384).  Its MMAs run in order, so S_t of the next key tile is issued right behind the product that
// reads p from the same columns.  A wait costs it some 200 clocks even where it is over, more than the MMAs behind it take
// to issue: a key tile has one barrier, and the second tile does not wait for keys again.  Shared memory: both query
// tiles, a ring of 16 KB key blocks (128 keys x 64 entries), a ring of value tiles.
//
// A block's instructions have to be fetched, some 16 clocks each the first time, so code is short where that costs
// little: masks are bit tests in a loop of their own, the capped softmax is a loop over 32 columns.  (Uncapped scores stay in
// registers: reloading them from TMEM 32 columns at a time took 2.59 ms at 1 x 16384.)
//
// Blocks stay: each takes over the grid's tiles that have not started yet (cluster launch control), so that the next
// item's queries and keys arrive during the last softmax and the output of the item before.  The grid's order is
// the order of the work: levels of query tiles, the longest first.  (A launch of a few tiles has no pairs: see pick_mode.)
// Every wait on an mbarrier is bounded; after one that runs out the block raises the device error word and leaves.  The meetings of two warps
// (barrier.cta.sync) end because a warp that leaves early arrives once more on its way out.
#pragma once
#include "zp_tc.cuh"

namespace zp {
namespace attn {

using namespace tc;

// registers of the feeding group's threads and of the others': 72 + 2 x 216 = 3 x 168 at launch, 56 + 4 x 104 <= 5 x 96
constexpr int threads_of(int groups) { return 128 + 256 * groups; }
constexpr int feed_regs(int groups) { return groups == 1 ? 72 : 56; }
constexpr int softmax_regs(int groups) { return groups == 1 ? 216 : 104; }
constexpr int BLK = 16384;               // 128 rows x 64 elements x 2 bytes
constexpr int NBAR = 8;                  // barriers of a ring, more than tiles in flight
constexpr uint32_t O_COL = 256;          // TMEM columns: S_0 | S_1 | O_0 | O_1, 128 each
constexpr int SLACK = 128;               // alignment padding that the launch provides for
constexpr float LOG2E = 1.4426950408889634f;

// Two tiles of one sequence.
struct Item {
  int b, head[2], hk;                    // sequence, query head of each tile, key/value head
  int q0[2], rows[2], pos[2];            // first row of q (absolute), rows, position of the first row
  int keys;                              // keys of the sequence: rows past them are not read
  int n[2];                              // key tiles 0 .. n - 1 of each
  int kept, t0;                          // key tile j is number j < kept ? j : t0 + j - kept
  bool real;                             // false: no more work
  __device__ __forceinline__ int most() const { return max(n[0], n[1]); }
  __device__ __forceinline__ int key0(int j) const { return (j < kept ? j : t0 + j - kept) * 128; }
};
struct __align__(16) Shared {
  uint4 work;                            // answer of cluster launch control
  Item item[2];                          // what the producer found, for the other roles
  uint64_t wfull, ifull[2], iempty[2], qfull, qempty, kfull[NBAR], kempty[NBAR], vfull[NBAR], vempty[NBAR], sfull[2], pfull[2][2], pvdone[2];
  float rows[2][2][128];                 // of the column halves of each tile: a step's maxima, an item's sums
  uint32_t tmem_base;
  int abort_flag;
};

// How a kernel's tiles share items.
enum { PAIR_HEADS = 0, PAIR_ROWS = 1, SINGLE = 2 };      // two heads of a key/value head, two row blocks of a head, no second tile
__device__ __forceinline__ int level_rows(int mode) { return mode == PAIR_ROWS ? 256 : 128; }
__device__ __forceinline__ int item_head(int mode, int x, int t) { return mode == PAIR_HEADS ? 2 * x + t : x; }
__device__ __forceinline__ int item_row(int mode, int first, int t) { return mode == PAIR_ROWS ? first + t * 128 : first; }
__device__ __forceinline__ int item_rows(int mode, int rows, int t) { return mode == SINGLE && t ? 0 : min(128, rows); }
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

// ---- masks and waits ---------------------------------------------------------------------------------
// the lowest n bits, n from below 0 to above 32
__device__ __forceinline__ uint32_t low_bits(int n) { return n <= 0 ? 0u : n >= 32 ? 0xffffffffu : (1u << n) - 1u; }
// The factor of the raw products as a positive number and what is left of it: masked products become -inf before they meet the factor.
struct Factor {
  float mag, sign;
  __device__ __forceinline__ explicit Factor(float s) : mag(s > 0.f || s < 0.f ? fabsf(s) : 1.f), sign(s > 0.f ? 1.f : s < 0.f ? -1.f : s) {}
};

// What P has to bring:
//   T                            element type;  SPLIT: weights as hi + lo (T = bf16);  MASKED: rows have a first visible key too
//   GROUPS                       groups of softmax warps a tile: 1, or 2 (CAPPED: 2)
//   LAZY                         powers of two by which a score may exceed its row's reference;  CAPPED: the reference is fixed
//   rings, error_word            members
//   item(id, it)                 the work of block `id`; false: none
//   prefetch()                   of its tensor maps
//   load_q(dst, bar, it, t)      TMA loads of a query tile;  Step(p, it, key0): where a key tile lies, and with it
//   load_k(dst, bar, it, step, i), load_v(dst, bar, it, step, i): TMA loads of one block each
//   Row(p, it, t, r)             one query row, with lim (last visible key) and, where MASKED, lo and keep (keys j < lo are not seen
//                                unless j < keep), ref0 (first reference; -inf unless CAPPED), and
//     fac                        what a raw product is multiplied by to become the exponent of 2 (its magnitude by the pipeline, or by
//     transform(s, key0)         (P::BIASED) that makes exponents of 2 of the raw products of 32 keys), or
//     weights4(s, w)             (CAPPED) four raw products to four weights
//     finish(p, ref, l)          factor of the row's sums (1 / l, gates)
//     entries(p, c, v)           (P::GATED) factors of 32 entries
//   out(row, head, c), dv        address of entry c of a row, entries of a head
template <class P>
__global__ void __launch_bounds__(threads_of(P::GROUPS), 1) attn_tc_kernel(const __grid_constant__ P p) {
  using T = typename P::T;
  constexpr int GROUPS = P::GROUPS, COLS = 128 / GROUPS, CHUNKS = COLS / 32;      // columns of a group
  constexpr int UNIT = 64 / GROUPS;      // keys that a group hands over at a time
  constexpr bool LATE = GROUPS == 1 && !P::SPLIT;      // the first of them behind half of the second's exponentials
  static_assert(GROUPS == 2 || !P::CAPPED, "capped scores come in halves of a row");
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
      mbar_init(&sh.ifull[i], 1); mbar_init(&sh.iempty[i], 1 + 8 * GROUPS);
      mbar_init(&sh.sfull[i], 1); mbar_init(&sh.pvdone[i], 1);
      for (int u = 0; u < 2; ++u) mbar_init(&sh.pfull[i][u], 4 * GROUPS);
    }
    mbar_init(&sh.wfull, 1); mbar_init(&sh.qfull, 1);
    mbar_init(&sh.qempty, 1);
    for (int i = 0; i < NBAR; ++i) {
      mbar_init(&sh.kfull[i], 1); mbar_init(&sh.kempty[i], 1);
      mbar_init(&sh.vfull[i], 1); mbar_init(&sh.vempty[i], 1);
    }
    sh.abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    if (lane == 0) p.prefetch();
    tmem_alloc(&sh.tmem_base, 512);
    tmem_relinquish();
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = sh.tmem_base;
  volatile int* abortp = &sh.abort_flag;
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(feed_regs(GROUPS)));
    if (warp == 0) {
      if (elect_one()) {
        // ---------------- work and loads ----------------
        Item it;
        dim3 id(blockIdx.x, blockIdx.y, blockIdx.z);
        uint32_t tiles = 0, kslot = 0, vslot = 0, nq = 0, asked = 0;      // key (value) tiles so far, next block (tile) of the rings
        uint32_t kfree = g.nk, kfreed = 0, vfreed = 0;                    // free key blocks, key and value tiles given back
        bool ok = true;
        ask_work(&sh.work, &sh.wfull);
        // the next block of the grid; every answer that was asked for is waited for, and a refusal is the last one
        auto next = [&]() -> bool {
          ok = mbar_wait(&sh.wfull, asked & 1, abortp, p.error_word, 821);
          ++asked;
          if (!ok || !read_work(&sh.work, id)) return false;
          ask_work(&sh.work, &sh.wfull);
          return true;
        };
        it.real = true;
        for (uint32_t w = 0; ok && it.real; ++w) {
          it.real = p.item(id, it);
          while (!it.real && next()) it.real = p.item(id, it);
          if (!ok || !mbar_wait<true>(&sh.iempty[w & 1], ((w >> 1) & 1) ^ 1, abortp, p.error_word, 822)) break;
          sh.item[w & 1] = it;
          mbar_arrive(&sh.ifull[w & 1]);
          if (!it.real) break;
          if (it.most() > 0) {
            ok = mbar_wait<true>(&sh.qempty, (nq & 1) ^ 1, abortp, p.error_word, 823);
            if (!ok) break;
            mbar_arrive_expect_tx(&sh.qfull, (uint32_t)(((it.n[0] > 0) + (it.n[1] > 0)) * g.nbq * BLK));
#pragma unroll
            for (int t = 0; t < 2; ++t)
              if (it.n[t] > 0) p.load_q(qbuf + t * g.nbq * BLK, &sh.qfull, it, t);
            ++nq;
          }
          for (int j = 0; ok && j < it.most(); ++j, ++tiles) {
            const typename P::Step step(p, it, it.key0(j));
            uint64_t* bar = &sh.kfull[tiles % NBAR];
            mbar_arrive_expect_tx(bar, (uint32_t)(g.nbq * BLK));
            for (int i = 0; ok && i < g.nbq; ++i) {
              if (kfree == 0) {                            // the oldest key tile's blocks
                ok = mbar_wait<true>(&sh.kempty[kfreed % NBAR], (kfreed / NBAR) & 1, abortp, p.error_word, 824);
                ++kfreed;
                kfree += g.nbq;
                if (!ok) break;
              }
              --kfree;
              p.load_k(kring + kslot * BLK, bar, it, step, i);
              if (++kslot == (uint32_t)g.nk) kslot = 0;
            }
            if (ok && tiles - vfreed == (uint32_t)g.nv) {
              ok = mbar_wait<true>(&sh.vempty[vfreed % NBAR], (vfreed / NBAR) & 1, abortp, p.error_word, 825);
              ++vfreed;
            }
            if (!ok) break;
            bar = &sh.vfull[tiles % NBAR];
            mbar_arrive_expect_tx(bar, (uint32_t)(g.nbv * BLK));
            for (int i = 0; i < g.nbv; ++i) p.load_v(vring + (vslot * g.nbv + i) * BLK, bar, it, step, i);
            if (++vslot == (uint32_t)g.nv) vslot = 0;
          }
          if (ok && !next()) it.real = false;
          if (ok && !it.real) {                            // tell the others, and leave
            ++w;
            if (mbar_wait<true>(&sh.iempty[w & 1], ((w >> 1) & 1) ^ 1, abortp, p.error_word, 826)) {
              sh.item[w & 1].real = false;
              mbar_arrive(&sh.ifull[w & 1]);
            }
          }
        }
      }
    } else if (warp == 1) {
      if (elect_one()) {
        // ---------------- products ----------------
        constexpr uint32_t ID_S = idesc_f16(UmmaFmt<T>::fmt, 128, 128);
        const uint32_t id_o = idesc_f16(UmmaFmt<T>::fmt, 128, 64 * g.nbv) | (1u << 16);      // V is MN-major
        const uint32_t q_addr = smem_u32(qbuf), k_addr = smem_u32(kring), v_addr = smem_u32(vring);
        uint32_t tiles = 0, cnt[2] = {0, 0}, kslot = 0, vslot = 0, nq = 0;      // key tiles of the items before, steps of each tile, places in the rings
        bool ok = true;
        for (uint32_t w = 0; ok; ++w) {
          ok = mbar_wait(&sh.ifull[w & 1], (w >> 1) & 1, abortp, p.error_word, 827);
          const int n[2] = {sh.item[w & 1].n[0], sh.item[w & 1].n[1]}, most = max(n[0], n[1]);
          if (!ok || !sh.item[w & 1].real) break;
          mbar_arrive(&sh.iempty[w & 1]);
          if (most <= 0) continue;
          ok = mbar_wait(&sh.qfull, nq & 1, abortp, p.error_word, 828);
          ++nq;
          // S of key tile j, whose blocks start at kslot; the last tile that reads it gives them back
          auto issue_s = [&](int t, int j) {
            const bool last = t == (j < n[1] ? 1 : 0);
            uint32_t slot = kslot;
#pragma unroll 1
            for (int i = 0; i < g.nbq; ++i) {
              const uint64_t ad = smem_desc_sw128(q_addr + (t * g.nbq + i) * BLK), bd = smem_desc_sw128(k_addr + slot * BLK);
#pragma unroll
              for (int c = 0; c < 4; ++c) umma_f16(tmem + t * 128, ad + 2u * c, bd + 2u * c, ID_S, (i | c) ? 1u : 0u);
              if (++slot == (uint32_t)g.nk) slot = 0;
            }
            umma_commit(&sh.sfull[t]);
            if (!last) return;
            umma_commit(&sh.kempty[(tiles + j) % NBAR]);
            kslot = slot;
            if (j == most - 1) umma_commit(&sh.qempty);
          };
          auto keys = [&](int j) -> bool {
            const bool in = mbar_wait(&sh.kfull[(tiles + j) % NBAR], ((tiles + j) / NBAR) & 1, abortp, p.error_word, 829);
            fence_after_sync();
            return in;
          };
          ok = ok && keys(0);
#pragma unroll
          for (int t = 0; t < 2; ++t)
            if (ok && n[t] > 0) issue_s(t, 0);
#pragma unroll 1
          for (int j = 0; ok && j < most; ++j) {
            const uint32_t k = tiles + j, v0 = v_addr + vslot * g.nbv * BLK;
            ok = mbar_wait(&sh.vfull[k % NBAR], (k / NBAR) & 1, abortp, p.error_word, 830);
#pragma unroll
            for (int t = 0; t < 2; ++t) {
              if (!ok || j >= n[t]) continue;
              const uint32_t pt = tmem + t * 128, ot = tmem + O_COL + t * 128;
#pragma unroll
              for (int u = 0; u < 2; ++u) {                  // the softmax hands over 64 keys at a time
                // (an item's first product overwrites all of O: every softmax warp of the tile is past the item before, whose output it read there)
                ok = ok && mbar_wait(&sh.pfull[t][u], cnt[t] & 1, abortp, p.error_word, 831);
                if (!ok) continue;
                fence_after_sync();
#pragma unroll
                for (int c = 0; c < 4; ++c) {                // 16 keys a step: 8 columns of p
                  const int key16 = GROUPS == 2 ? (c >> 1) * 4 + 2 * u + (c & 1) : 4 * u + c;
                  const uint64_t bd = smem_desc_mn(v0 + key16 * 2048);
                  const uint32_t a = pt + (key16 >> 1) * 32 + (key16 & 1) * 8;
                  umma_ts(ot, a, bd, id_o, (j | u | c) ? 1u : 0u);
                  if (P::SPLIT) umma_ts(ot, a + 16, bd, id_o, 1u);
                }
              }
              if (!ok) continue;
              ++cnt[t];
              // (before the next scores are reported: the softmax's wait compares parities, and after those scores it could otherwise
              // take the product two steps back for the last one)
              umma_commit(&sh.pvdone[t]);
              if (j + 1 < n[t]) {                            // (behind the product that reads p from its columns)
                if (t == 0 || j + 1 >= n[0]) ok = keys(j + 1);
                if (ok) issue_s(t, j + 1);
              }
            }
            if (ok) umma_commit(&sh.vempty[k % NBAR]);
            if (++vslot == (uint32_t)g.nv) vslot = 0;
          }
          tiles += most;
        }
      }
    }
  } else {
    // ---------------- softmax ----------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(softmax_regs(GROUPS)));
    const int grp = (warp - 4) >> 2, t = grp / GROUPS, half = grp % GROUPS, quad = warp & 3;      // tile, its columns, TMEM lane quadrant
    const int r = quad * 32 + lane;                                                              // row of the tile
    const uint32_t lanes = tmem + (static_cast<uint32_t>(quad * 32) << 16), st = lanes + t * 128, ot = lanes + O_COL + t * 128;
    // Meeting of the two warps with the same rows; false: the block is giving up.  (A warp that leaves early arrives once more: the other one
    // can be at one meeting at most before it sees the abort flag, which was raised before.)
    const int pair = 1 + t * 4 + quad;
    auto meet = [&]() -> bool {
      asm volatile("barrier.cta.sync %0, 64;" ::"r"(pair) : "memory");
      return __all_sync(0xffffffffu, !*abortp);
    };
    uint32_t tiles = 0, cnt = 0, vslot = 0;      // key tiles of the items before, steps of this tile, place in the value ring
    bool ok = true;
    for (uint32_t w = 0; ok; ++w) {
      ok = mbar_wait_warp(&sh.ifull[w & 1], (w >> 1) & 1, abortp, p.error_word, 832);
      if (!ok || !sh.item[w & 1].real) break;
      const Item it = sh.item[w & 1];
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.iempty[w & 1]);
      const int n = of_tile(it.n, t), most = it.most();
      const typename P::Row row(p, it, t, r);
      float2 l2 = make_float2(0.f, 0.f);
      float ref = row.ref0;
      // A block's first turn works on nothing (step -1: no waits, no stores): it fetches the loop's instructions while the first
      // operands are on their way, which otherwise come one after the other behind them (5 to 11 thousand clocks).
      for (int j = w == 0 ? -1 : 0; ok && j < n; ++j) {
        const bool dry = j < 0;
        const int key0 = it.key0(j) + half * COLS;      // first key of this group
        if (!dry) ok = mbar_wait_warp(&sh.sfull[t], cnt & 1, abortp, p.error_word, 833);
        if (!ok) break;
        fence_after_sync();
        bool whole = key0 + COLS - 1 <= row.lim;
        if constexpr (P::MASKED) whole = whole && (key0 >= row.lo || key0 + COLS <= row.keep);
        if constexpr (!P::CAPPED) whole = whole && row.fac.sign == 1.f;
        whole = __all_sync(0xffffffffu, whole || dry);
        auto seen = [&](int key) -> uint32_t {          // of 32 keys
          uint32_t m = low_bits(row.lim - key + 1);
          if constexpr (P::MASKED) m &= ~low_bits(row.lo - key) | low_bits(row.keep - key);
          return m;
        };
        // UNIT keys' weights are written.  Value rows past the sequence become zeros (0 times another sequence's values could be
        // NaN): those that the product behind this hand-over reads, whichever tile's comes first
        auto hand_over = [&](int u) {
          if (dry) return;
          const int first = half * COLS + UNIT * u, left = max(it.keys - it.key0(j) - first, 0);
          if (left < UNIT) {
            const uint32_t k = tiles + j;
            ok = mbar_wait_warp(&sh.vfull[k % NBAR], (k / NBAR) & 1, abortp, p.error_word, 835);
#pragma unroll 1
            for (int i = r; ok && i < (UNIT - left) * 8 * g.nbv; i += 128) {
              const int line = i >> 3, blk = line / (UNIT - left), key = first + left + line % (UNIT - left);
              *reinterpret_cast<int4*>(vring + (vslot * g.nbv + blk) * BLK + key * 128 + ((i & 7) << 4)) = make_int4(0, 0, 0, 0);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          }
          tmem_st_wait();
          fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.pfull[t][u]);
        };
        // weights of 32 keys, over their scores: hi in the first 16 columns, lo in the others
        auto weights = [&](uint32_t (&s)[32], int c, float mref) {
          const uint32_t y = P::CAPPED && !whole ? seen(key0 + c) : 0xffffffffu, at = st + half * COLS + c;
          uint32_t hi[16], lo[16];
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            float wt[4];
            if constexpr (P::CAPPED) {
              row.weights4(&s[i], wt);
              if (!whole) {
#pragma unroll
                for (int u = 0; u < 4; ++u)
                  if (!(y >> (i + u) & 1u)) wt[u] = 0.f;
              }
            } else {
              const float sc = P::BIASED ? 1.f : row.fac.mag;
#pragma unroll
              for (int u = 0; u < 4; u += 2) {
                float2 x = make_float2(-mref, -mref);
                ffma2(x, make_float2(__uint_as_float(s[i + u]), __uint_as_float(s[i + u + 1])), make_float2(sc, sc));
                wt[u] = ex2_approx(x.x);
                wt[u + 1] = ex2_approx(x.y);
              }
            }
            l2 = fadd2(l2, fadd2(make_float2(wt[0], wt[1]), make_float2(wt[2], wt[3])));
#pragma unroll
            for (int u = 0; u < 4; u += 2) {
              const float2 w2 = make_float2(wt[u], wt[u + 1]);
              if constexpr (P::SPLIT && P::CAPPED) {         // (rounded in fp32 the upper parts need no unpacking)
                const float2 f = round8(w2), rest = fsub2(w2, f);
                hi[(i + u) >> 1] = upper_halves(f);
                const typename Pair<T>::V z = Pair<T>::pack(rest.x, rest.y);
                lo[(i + u) >> 1] = *reinterpret_cast<const uint32_t*>(&z);
                continue;
              }
              const typename Pair<T>::V x = Pair<T>::pack(w2.x, w2.y);
              hi[(i + u) >> 1] = *reinterpret_cast<const uint32_t*>(&x);
              if constexpr (P::SPLIT) {
                const float2 rest = fsub2(w2, Pair<T>::unpack(x));
                const typename Pair<T>::V z = Pair<T>::pack(rest.x, rest.y);
                lo[(i + u) >> 1] = *reinterpret_cast<const uint32_t*>(&z);
              }
            }
          }
          if (LATE && c == 64) hand_over(0);
          if (dry) return;
          tmem_st16(at, hi);
          if constexpr (P::SPLIT) tmem_st16(at + 16, lo);
        };
        if constexpr (P::CAPPED) {
#pragma unroll 1
          for (int c = 0; c < COLS; c += 32) {
            uint32_t s[32];
            tmem_ld32_issue(st + half * COLS + c, s);
            tmem_ld32_wait(s);
            weights(s, c, 0.f);
            hand_over(c >> 5);
          }
        } else {
          const uint32_t at = st + half * COLS;
          if (!whole) {
#pragma unroll 1
            for (int c = 0; c < COLS; c += 32) {
              uint32_t s[32];
              tmem_ld32_issue(at + c, s);
              const uint32_t y = seen(key0 + c);
              tmem_ld32_wait(s);
              if (row.fac.sign != 1.f) {                     // (a factor that is negative or zero)
#pragma unroll
                for (int i = 0; i < 32; ++i) s[i] = __float_as_uint(__uint_as_float(s[i]) * row.fac.sign);
              }
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (!(y >> i & 1u)) s[i] = 0xff800000u;      // -inf
              tmem_st32(at + c, s);
            }
            tmem_st_wait();
          }
          uint32_t s[CHUNKS][32];
          float m[CHUNKS];
          if constexpr (GROUPS == 1) {
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) tmem_ld32_issue(at + c * 32, s[c]);
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) tmem_ld32_wait(s[c]);
          } else {
            tmem_ld32_issue(at, s[0]);
            tmem_ld32_wait(s[0]);
            tmem_ld32_issue(at + 32, s[1]);      // (on its way while the first part is compared)
          }
#pragma unroll
          for (int c = 0; c < CHUNKS; ++c) {
            if (GROUPS == 2 && c == 1) tmem_ld32_wait(s[1]);
            if constexpr (P::BIASED) row.transform(s[c], key0 + c * 32);
            m[c] = fmaxf(__uint_as_float(s[c][0]), __uint_as_float(s[c][1]));
#pragma unroll
            for (int i = 2; i < 32; i += 2) m[c] = fmax3(m[c], __uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1]));
          }
#pragma unroll
          for (int c = 1; c < CHUNKS; ++c) m[0] = fmaxf(m[0], m[c]);
          if constexpr (!P::BIASED) m[0] *= row.fac.mag;
          if (GROUPS == 2 && !dry) {                         // the row's maximum is that of both halves
            sh.rows[t][half][r] = m[0];
            ok = meet();
            if (!ok) break;
            m[0] = fmaxf(m[0], sh.rows[t][half ^ 1][r]);
          }
          const bool moves = !dry && m[0] > ref + P::LAZY;
          if (__any_sync(0xffffffffu, moves)) {              // (the same rows and the same answer in both halves' warps)
            const float fac = moves ? ex2_approx(ref - m[0]) : 1.f;
            if (moves) ref = m[0];
            l2.x *= fac;
            l2.y *= fac;
            if (j > 0) {
              ok = mbar_wait_warp(&sh.pvdone[t], (cnt & 1) ^ 1, abortp, p.error_word, 834);
              if (!ok) break;
              fence_after_sync();
#pragma unroll 1
              for (int c = 16 * half; c < 64 * g.nbv; c += 16 * GROUPS) {
                uint32_t o[16];
                tmem_ld16(ot + c, o);
#pragma unroll
                for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * fac);
                tmem_st16(ot + c, o);
              }
              // (Nothing hangs on this meeting: the product waits for every warp's weights, which are handed over behind its own stores.  But the
              // code without it is the slower one: latents of 3 x 600 to 3000 tokens 360 -> 367 us, 2 x 500 to 1500 154 -> 156.)
              if constexpr (GROUPS == 2) {
                tmem_st_wait();
                fence_before_sync();
                ok = meet();
                if (!ok) break;
                fence_after_sync();
              }
            }
          }
          const float mref = ref == -INFINITY ? 0.f : ref;      // (no key seen so far: every weight is exp2(-inf))
#pragma unroll
          for (int c = 0; c < CHUNKS; ++c) {
            weights(s[c], c * 32, mref);
            if (GROUPS == 2) hand_over(c);
            else if (LATE ? c == 3 : c & 1) hand_over(c >> 1);
          }
        }
        if (dry) {
          l2 = make_float2(0.f, 0.f);
          continue;
        }
        ++cnt;
        if (++vslot == (uint32_t)g.nv) vslot = 0;
      }
      if (!ok) break;
      vslot = (vslot + most - n) % g.nv;
      tiles += most;
      // ---- output: four lanes share a row's 64 bytes ----
      float l = l2.x + l2.y;
      if (n > 0) {
        ok = mbar_wait_warp(&sh.pvdone[t], (cnt & 1) ^ 1, abortp, p.error_word, 836);
        if (!ok) break;
        fence_after_sync();
        if constexpr (GROUPS == 2) {      // (the last product waited for both halves' weights, and with them for their reads of the other's maximum)
          sh.rows[t][half][r] = l;
          ok = meet();
          if (!ok) break;
          l = sh.rows[t][0][r] + sh.rows[t][1][r];
          ok = meet();                                       // (the next step's maxima go to the same place)
          if (!ok) break;
        }
      }
      const float inv = row.finish(p, ref, l);
      const int rows = of_tile(it.rows, t), q0 = of_tile(it.q0, t), head = of_tile(it.head, t), r4 = r & ~3, c8 = (lane & 3) * 8;
#pragma unroll 1
      for (int c = half * 32; c < 64 * g.nbv; c += 32 * GROUPS) {
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
      fence_before_sync();      // (the next item's first product into O follows the next arrival of every softmax warp of this tile)
    }
    if (GROUPS == 2 && !ok) asm volatile("barrier.cta.arrive %0, 64;" ::"r"(pair) : "memory");
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
static_assert(14 * BLK + SLACK + sizeof(Shared) <= 232448, "14 blocks of operands");
static inline Rings rings_of(int nbq, int nbv) {
  const int blocks = (232448 - SLACK - (int)sizeof(Shared)) / BLK - 2 * nbq;
  Rings g{nbq, nbv, 0, nbq > 3 ? 1 : 2};
  g.nk = blocks - g.nv * nbv;
  if (g.nk > (NBAR - 1) * nbq) g.nk = (NBAR - 1) * nbq;
  return g;
}

// The most 128-row query tiles that the sequences can have, all heads (the counts are on the device).
static inline int64_t most_tiles(int heads, int B, int total_q, int max_q) {
  const int64_t by_rows = (int64_t)total_q / 128 + B, by_longest = (int64_t)B * ((max_q + 127) / 128);
  return heads * (by_rows < by_longest ? by_rows : by_longest);
}
// Pairs, unless every tile can have an SM to itself: a launch that short is one tile's latency, which the second tile of a pair only adds to.
// Prompts, single tiles / pairs: 1 x 100 tokens, 32 heads: 10.3 / 12.1 us; 4 of up to 400, 8 heads: 20.3 / 22.1; 16 of up to 100,
// 16 heads (256 tiles): 51.5 / 32.5.  (One query tile a block with a pass for the maxima and one for the weights, as it was before, had all its softmax
// warps on that tile: at up to 148 tiles it took 0 to 3 us less of 10 to 30, from there on 1.2 to 3.5 times as long.)
// (Measured with one group of softmax warps; two for few keys take up to 0.4 us off a single tile.  Windows and latents of few tiles have
// kernels of their own, and no single tiles here.)
static inline int pick_pair(int heads_per_kv) { return heads_per_kv % 2 == 0 ? PAIR_HEADS : PAIR_ROWS; }
static inline int pick_mode(int heads, int heads_per_kv, int B, int total_q, int max_q) {
  return most_tiles(heads, B, total_q, max_q) <= 148 ? SINGLE : pick_pair(heads_per_kv);
}
static inline dim3 grid_of(int mode, int heads, int B, int max_q, int& levels) {
  const int rows = mode == PAIR_ROWS ? 256 : 128;
  levels = (max_q + rows - 1) / rows;
  return dim3(mode == PAIR_HEADS ? heads / 2 : heads, B, levels);
}

template <class P>
static int launch_attn(const P& p, dim3 grid, cudaStream_t st, const char* what) {
  const int smem = (2 * p.rings.nbq + p.rings.nk + p.rings.nv * p.rings.nbv) * BLK + (int)sizeof(Shared) + SLACK;
  cudaError_t e = cudaFuncSetAttribute(attn_tc_kernel<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) { set_error("%s: %s", what, cudaGetErrorString(e)); return ZP_ERR_CUDA; }
  attn_tc_kernel<P><<<grid, threads_of(P::GROUPS), smem, st>>>(p);
  return check_launch(what);
}

}  // namespace attn
}  // namespace zp

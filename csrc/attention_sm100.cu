// Flash attention for sm_100a (head_dim 128, bf16): tcgen05 QKᵀ / PV with TMEM accumulators, TMA-staged operands,
// online softmax with one thread per query row.  Role parity: reference kernels/flash_attn.py:162-212
// (nki_flash_attn_func → flash_fwd / flash_attn_bwd) and modules/attention call sites.
//
// Forward, persistent, one CTA per SM walking items of 256 query rows of one (head, batch): two 128-row tiles that share every
// K / V tile and are half a step out of phase, so that one tile's softmax runs under the other tile's products.
// TMEM (512 columns): S of tile 0 / 1, O of tile 0 / 1, 128 columns each.
//   warps 0-3, 4-7  softmax  : thread = query row of tile 0 / 1 (tcgen05.ld 32x32b: lane ↔ TMEM lane): row max, exp2, row sum, P
//                              packed to bf16 and written back over S with tcgen05.st.  The O accumulator is only rescaled when
//                              the running max grew by more than 2^8 (lazy rescale), so the common tile does no TMEM
//                              round trip for O at all.
//   warps 8-11  output       : O of a finished tile out of TMEM, divided by the row sums, to memory, while the softmax goes on to the next item
//   warp 12     TMA producer : Q0, Q1, then K_j / V_j tiles ([128 kv × 128 d] as two 128B-swizzled [128 × 64] boxes), ring of 4
//   warp 13     MMA issuer   : S = Q·K_jᵀ  (A, B K-major, 8 × UMMA 128×128×16)
//                              O += P·V_j (A = P read from TMEM, B = V MN-major)
// Outputs: O (bf16, arbitrary b/s/h strides) and LSE (fp32 [B, H, S], natural log) for the backward.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <string>

#include "common.cuh"
#include "kernels.h"
#include "sm100_ptx.cuh"

namespace nxd {

CUtensorMap make_tmap_bf16_heads(const void* ptr, const uint64_t (&dims)[4], const uint64_t (&strides)[3], uint32_t box_cols, uint32_t box_rows);

namespace fa {

constexpr int BM = 128, BN = 128, HD = 128;
constexpr int kThreads = 512;
constexpr int kRing = 4;                         // K / V tiles in flight or in use
constexpr uint32_t kTile = BM * HD * 2;          // 32 KB
constexpr uint32_t kHalf = kTile / 2;            // one [128 × 64] box
constexpr uint32_t kStage = 32 * 64 * 2;         // an output warp's 32 rows x 64 columns on their way to memory
constexpr uint32_t kSmemFwd = (2 + kRing) * kTile + 4 * kStage + 2048 /*row sums*/ + 1024 /*align*/ + 512 /*barriers*/;

// Warp-uniform issue: the whole MMA warp runs the issue loop in convergent control flow and one elected lane executes the tcgen05
// instructions (sm100_ptx.cuh explains why).  One election serves the products of a whole tile and the barrier they complete; descriptors
// advance by constants.  With an election, a predicate and a new descriptor for each product the issuing warp was what a backward step
// waited for: 32 products of 32 to 64 cycles took it 2200 cycles.
#define NXD_FA_MMA "@q tcgen05.mma.cta_group::1.kind::f16 "
#define NXD_FA_BEGIN                                                                                                     \
  "{\n\t.reg .pred p, q, t;\n\t.reg .b64 a, b;\n\t.reg .b32 c;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t" \
  "setp.eq.b32 t, 0, 0;\n\t"
#define NXD_FA_COMMIT(bar) "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [" bar "];\n\t"
#define NXD_FA_SS(ia, ib) "add.s64 a, %1, " ia ";\n\tadd.s64 b, %2, " ib ";\n\t" NXD_FA_MMA "[%0], a, b, %3, t;\n\t"
#define NXD_FA_TS(ia, ib) "add.u32 c, %1, " ia ";\n\tadd.s64 b, %2, " ib ";\n\t" NXD_FA_MMA "[%0], [c], b, %3, t;\n\t"
// Eight products over 128 elements of K, both operands in shared memory; product i reads (i / 4) * 4 and (i % 4) * 1 steps (of 16 bytes) on.
template <int A4, int A1, int B4, int B1>
NXD_DEVICE void mma_ss8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, uint32_t bar) {
  asm volatile(NXD_FA_BEGIN NXD_FA_MMA "[%0], %1, %2, %3, p;\n\t"
               NXD_FA_SS("%6", "%13") NXD_FA_SS("%7", "%14") NXD_FA_SS("%8", "%15") NXD_FA_SS("%9", "%16") NXD_FA_SS("%10", "%17")
               NXD_FA_SS("%11", "%18") NXD_FA_SS("%12", "%19") NXD_FA_COMMIT("%5") "}"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(bar),
                 "n"(A1), "n"(2 * A1), "n"(3 * A1), "n"(A4), "n"(A4 + A1), "n"(A4 + 2 * A1), "n"(A4 + 3 * A1),
                 "n"(B1), "n"(2 * B1), "n"(3 * B1), "n"(B4), "n"(B4 + B1), "n"(B4 + 2 * B1), "n"(B4 + 3 * B1)
               : "memory");
}
// Four products over 64 elements of K, A in TMEM (P of the forward, Pᵀ and dSᵀ of the backward); the last two read A from A2 columns on.
template <int A2, int B1>
NXD_DEVICE void mma_ts4(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(NXD_FA_BEGIN NXD_FA_MMA "[%0], [%1], %2, %3, p;\n\t" NXD_FA_TS("8", "%5") NXD_FA_TS("%8", "%6") NXD_FA_TS("%9", "%7") "}"
               ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate), "n"(B1), "n"(2 * B1), "n"(3 * B1), "n"(A2), "n"(A2 + 8)
               : "memory");
}
NXD_DEVICE void tcgen05_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
NXD_DEVICE void tcgen05_st_32x16p(uint32_t taddr, const uint32_t* r) {   // first 16 registers of a larger array
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
NXD_DEVICE void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
NXD_DEVICE void tcgen05_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
NXD_DEVICE void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
NXD_DEVICE void bulk_wait_read1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }
NXD_DEVICE void bulk_wait0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
NXD_DEVICE uint64_t pack2u(uint32_t a, uint32_t b) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b)); return r; }
NXD_DEVICE float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
NXD_DEVICE float max3_nan(float a, float b, float c) {       // NaN where one is
  float r;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
NXD_DEVICE uint32_t pack_bf16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// TMA coordinates of element (b, head, s, 0) in a map of dimensions (d, s, head, b): (0, s, head * h, b * b).  h, b: 1, or 0 where the view has one
// head or sequence, or repeats one (stride 0).
struct Coord { int h, b; };

struct FwdParams {
  int S_q, S_kv, H, Hkv, B;
  Coord q, k, v;
  long o_sb, o_ss, o_sh;      // output strides in elements
  float scale, scale_log2;
  int causal;
  int group_bh;               // (batch, head) pairs whose K / V stay in L2 together
  int split;                  // both streams on one query tile (see fwd_item)
  float* lse;                 // [B, H, S_q]
};

// Work items.  Two streams (t = 0, 1; a softmax warpgroup, an S and an O buffer each) share a block:
//   pair  : query tiles 2 qt, 2 qt + 1 of one (batch, head); both streams walk the same K / V tiles (causal: the second needs one
//           more; behind an odd number of tiles there is no second).
//   split : few tiles for many SMs (every block gets one item): both streams work on the SAME query tile, stream t takes the K / V
//           tiles of its parity and the partial results are merged at the end, which halves the serial chain.
// Items come heaviest first within groups of heads whose K / V stay in L2 together, and a block that is done takes the next one
// from the hardware's queue of blocks that have not started (cluster launch control): no counter in memory to clear.  All heads
// heaviest first made every block stream another head and re-read K / V from HBM for every tile; a fixed assignment left blocks idle for a fifth
// of the time (2 x 4096 tokens, 32 heads: 440 of 555 thousand cycles active).
struct FwdItem { int qt, head, b, n, n0, n1; };

NXD_DEVICE FwdItem fwd_item(int idx, const FwdParams& p) {
  FwdItem it{};
  if (idx < 0) return it;                          // n = 0: no item
  const int nq = (p.S_q + BM - 1) / BM, np = p.split ? nq : (nq + 1) / 2, bhs = p.H * p.B;
  const int grp = idx / (np * p.group_bh), rem = idx - grp * np * p.group_bh;
  const int gs = min(p.group_bh, bhs - grp * p.group_bh);
  const int bh = grp * p.group_bh + rem % gs, at = np - 1 - rem / gs;
  it.head = bh % p.H;
  it.b = bh / p.H;
  const int n_tiles_kv = (p.S_kv + BN - 1) / BN;
  if (p.split) {
    it.qt = at;
    it.n = p.causal ? min(at + 1, n_tiles_kv) : n_tiles_kv;
    it.n0 = (it.n + 1) / 2;
    it.n1 = it.n / 2;
  } else {
    it.qt = 2 * at;
    it.n0 = p.causal ? min(it.qt + 1, n_tiles_kv) : n_tiles_kv;
    it.n1 = it.qt + 1 >= nq ? 0 : p.causal ? min(it.qt + 2, n_tiles_kv) : n_tiles_kv;
    it.n = max(it.n0, it.n1);
  }
  return it;
}

// The block asks for the index of a block that has not started; the 16-byte answer completes `bar`.
NXD_DEVICE void clc_request(uint32_t answer, uint32_t bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(answer), "r"(bar) : "memory");
}
NXD_DEVICE int clc_answer(uint32_t answer) {       // block index, or -1: none left
  uint32_t got, x;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 h;\n\t"
      "ld.shared.b128 h, [%2];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "mov.u32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n\t}"
      : "=&r"(got), "=&r"(x)
      : "r"(answer)
      : "memory");
  return got ? (int)x : -1;
}

// P = 2^(s * scale - max) of 32 columns, packed to bf16 in their first half; `sum` grows by it.  MAX: the maximum of the whole row beside it, NaN
// where there is one.
template <bool MAX>
NXD_DEVICE void fwd_exps(uint32_t (&r)[4][32], int c, uint64_t scale, uint64_t shift, uint64_t& sum, float& mx) {
  float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    if constexpr (MAX) {
#pragma unroll
      for (int k = 0; k < 4; ++k) m4[k] = max3_nan(m4[k], __uint_as_float(r[k][i]), __uint_as_float(r[k][i + 1]));
    }
    const uint64_t x = fma2(pack2u(r[c][i], r[c][i + 1]), scale, shift);
    float p0, p1;
    unpack2(x, p0, p1);
    p0 = ex2(p0);
    p1 = ex2(p1);
    sum = add2(sum, pack2(p0, p1));
    r[c][i >> 1] = pack_bf16(p0, p1);
  }
  if constexpr (MAX) mx = max3_nan(m4[0], m4[1], max3_nan(m4[2], m4[3], m4[3]));
}
// columns behind `lim` to −inf: 0 after the exponential
NXD_DEVICE void fwd_mask(uint32_t (&r)[32], int lim) {
#pragma unroll
  for (int i = 0; i < 32; ++i)
    if (i > lim) r[i] = 0xff800000u;
}

// Bound by the tensor pipe and what feeds it: a tile's two products are 1024 cycles of mathematics and as many of operands and TMA writes in
// shared memory, and take about 1450.  Beside them go the exponentials (128 a row: 1024 cycles per tile and softmax warp, two warps per
// scheduler).  Tensor order is S0 S1 | PV0_j S0_{j+1} | PV1_j S1_{j+1} | …, across item boundaries, with one S buffer per stream: S_{j+1}
// follows PV_j in pipe order, so a softmax warp that sees S_{j+1} knows that PV_j is done.  Behind an item's first tile the exponentials begin with
// the maximum of the tiles before; the tile's own comes out beside the first quarter of them, which is done again where it lies more than 2^8
// above (maximum first: 1 x 8192, 32 heads, 457 us, so 449).  A warpgroup of its own for O: 1 x 1531, 64 heads on 8, 55.5 -> 49.3 us, 1 x 2048, 32
// heads 45.1 -> 41.1 with it and the next item's first product behind a stream's own last one.  Left out, none of them faster: P handed
// over in two or three parts, a quarter of the exponentials by polynomial.
__global__ void __launch_bounds__(kThreads, 1)
fa_fwd_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
              const __grid_constant__ CUtensorMap tv, __nv_bfloat16* __restrict__ out, const FwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sQ = smem_base, sKV = smem_base + 2 * kTile, sO = sKV + kRing * kTile, sStat = sO + 4 * kStage;
  const uint32_t bars = sStat + 2048;
  // per stream: qf[2] qe[2] s[2] p[2] of[2] oe[2] lf[2] le[2] | next item: full[2] empty[2] answer[2] | ring: kvf[] kve[] | tmem slot
  const uint32_t bar_qf = bars, bar_qe = bars + 16, bar_s = bars + 32, bar_p = bars + 48, bar_of = bars + 64,
                 bar_oe = bars + 80, bar_lf = bars + 96, bar_le = bars + 112, bar_nf = bars + 128, bar_ne = bars + 144, answers = bars + 160,
                 bar_kvf = bars + 192, bar_kve = bar_kvf + 8 * kRing, tmem_slot = bar_kve + 8 * kRing;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  auto load_q = [&](const FwdItem& it, int t) {
    const int qr = (it.qt + t) * BM, qh = it.head * p.q.h, qb = it.b * p.q.b;
    mbar_expect_tx(bar_qf + 8 * t, kTile);
    tma_load_4d(sQ + t * kTile, &tq, bar_qf + 8 * t, 0, qr, qh, qb);
    tma_load_4d(sQ + t * kTile + kHalf, &tq, bar_qf + 8 * t, 64, qr, qh, qb);
  };
  auto load_kv = [&](const CUtensorMap* map, int slot, int r, int h, int b) {
    mbar_expect_tx(bar_kvf + 8 * slot, kTile);
    tma_load_4d(sKV + slot * kTile, map, bar_kvf + 8 * slot, 0, r, h, b);
    tma_load_4d(sKV + slot * kTile + kHalf, map, bar_kvf + 8 * slot, 64, r, h, b);
  };
  if (warp == 12 && lane == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_qf + 8 * i, 1); mbar_init(bar_qe + 8 * i, 1); mbar_init(bar_s + 8 * i, 1);
      mbar_init(bar_p + 8 * i, 128); mbar_init(bar_of + 8 * i, 1); mbar_init(bar_oe + 8 * i, 128);
      mbar_init(bar_lf + 8 * i, 128); mbar_init(bar_le + 8 * i, 128);
      mbar_init(bar_nf + 8 * i, 1); mbar_init(bar_ne + 8 * i, 14);       // readers: softmax, output, producer and MMA warps
    }
    for (int i = 0; i < kRing; ++i) { mbar_init(bar_kvf + 8 * i, 1); mbar_init(bar_kve + 8 * i, 1); }
    fence_barrier_init();
    // the first item's Q and first K are on their way while the tensor memory is allocated
    const FwdItem it = fwd_item(blockIdx.x, p);
    const int kvh = it.head / (p.H / p.Hkv);
    load_q(it, 0);
    load_kv(&tk, 0, 0, kvh * p.k.h, it.b * p.k.b);
    if (it.n1 > 0 && !p.split) load_q(it, 1);
  }
  if (warp == 13) {
    tcgen05_alloc(tmem_slot, 512);
    tcgen05_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  const uint32_t tmem_S = tmem_base, tmem_O = tmem_base + 256;
  // item number il of this block (-1: none), for a whole warp or for the producer's lane alone
  auto item_index = [&](int il, bool whole_warp) {
    if (il == 0) return (int)blockIdx.x;
    if (p.split) return -1;                        // one item per block
    const int st = (il - 1) & 1;
    mbar_wait(bar_nf + 8 * st, (uint32_t)(((il - 1) >> 1) & 1));
    const int idx = clc_answer(answers + 16 * st);
    fence_async_smem();                            // this read before the next answer is written there
    if (whole_warp) __syncwarp();
    if (!whole_warp || lane == 0) mbar_arrive(bar_ne + 8 * st);
    return idx;
  };

  // registers: 128 a thread at launch, 2 x 168 + 88 + 88 = 4 x 128 from here on (nothing spills; 184, 80, 64 did: 1 x 600 tokens 22.7 us, so 20.7)
  if (warp >= 12) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    if (warp == 12 && lane == 0) {
      int slot = 0; uint32_t ph = 0;
      uint32_t q_items[2] = {0, 0};
      auto next = [&](const CUtensorMap* map, int r, int h, int b, bool loaded) {
        if (!loaded) {
          mbar_wait(bar_kve + 8 * slot, ph ^ 1);
          load_kv(map, slot, r, h, b);
        }
        if (++slot == kRing) { slot = 0; ph ^= 1; }
      };
      for (int il = 0;; ++il) {
        const int idx = item_index(il, false);
        if (idx < 0) break;
        const FwdItem it = fwd_item(idx, p);
        const int kvh = it.head / (p.H / p.Hkv);
        const int kh = kvh * p.k.h, kb = it.b * p.k.b, vh = kvh * p.v.h, vb = it.b * p.v.b;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (t == 0 || (it.n1 > 0 && !p.split)) {
            if (il > 0) {
              mbar_wait(bar_qe + 8 * t, (q_items[t] & 1) ^ 1);
              load_q(it, t);
            }
            ++q_items[t];
          }
          if (t == 0) next(&tk, 0, kh, kb, il == 0);
        }
        for (int j = 0; j < it.n; ++j) {
          if (j > 0) next(&tk, j * BN, kh, kb, false);
          next(&tv, j * BN, vh, vb, false);
        }
        // asked for when the last tile is on its way (two steps before the end): asked at the item's start, the blocks would share
        // out the queue before they know which of them are done first (1 x 2048 tokens, 32 heads: 59 us)
        if (!p.split) {
          mbar_wait(bar_ne + 8 * (il & 1), (uint32_t)(((il >> 1) & 1) ^ 1));
          mbar_expect_tx(bar_nf + 8 * (il & 1), 16);
          clc_request(answers + 16 * (il & 1), bar_nf + 8 * (il & 1));
        }
      }
    } else if (warp == 13) {
      // all 32 lanes run this loop; the helpers elect one lane
      constexpr uint32_t idesc_s = make_idesc(false, false, BM, BN);
      constexpr uint32_t idesc_o = make_idesc(false, true, BM, HD);
      uint32_t steps = 0, q_items = 0, o_items = 0;                  // bit t: parity of stream t's count
      // stream t, K tile number `pos` of the ring; `last_k`: no other stream uses it after this; `first` / `last` of the item
      auto issue_s = [&](int t, int pos, bool first, bool last, bool last_k) {
        const int slot = pos % kRing, tq_ = p.split ? 0 : t;
        if (first) { mbar_wait(bar_qf + 8 * tq_, (q_items >> t) & 1); q_items ^= 1u << t; }
        mbar_wait(bar_kvf + 8 * slot, (uint32_t)((pos / kRing) & 1));
        tcgen05_fence_after();
        mma_ss8<kHalf / 16, 2, kHalf / 16, 2>(tmem_S + t * BN, make_smem_desc(sQ + tq_ * kTile, 16, 1024), make_smem_desc(sKV + slot * kTile, 16, 1024),
                                              idesc_s, 0u, bar_s + 8 * t);
        if (last_k) tcgen05_commit_e(bar_kve + 8 * slot);
        if (last && !p.split) tcgen05_commit_e(bar_qe + 8 * t);
      };
      auto get = [&](int il) { return fwd_item(item_index(il, true), p); };
      // ring position of step j of stream t (its K; V is the next), counted from the item's first
      auto at = [&](int t, int j) { return p.split ? 2 * (2 * j + t) : 2 * j; };
      FwdItem it = get(0);
      int pos0 = 0;                                // ring position of the item's first K tile
      for (int t = 0; t < 2; ++t) {
        const int nt = t ? it.n1 : it.n0;
        if (nt > 0) issue_s(t, at(t, 0), true, nt == 1, p.split || t == 1 || it.n1 == 0);
      }
      for (int il = 0; it.n > 0; ++il) {
        FwdItem nx{};
        const int pos1 = pos0 + 2 * it.n, steps_n = max(it.n0, it.n1);
        bool asked = false;
        for (int j = 0; j < steps_n; ++j) {
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const int nt = t ? it.n1 : it.n0;
            if (j < nt) {
              const int pos = pos0 + at(t, j) + 1, slot = pos % kRing;
              const uint32_t ph = (steps >> t) & 1;
              steps ^= 1u << t;
              mbar_wait(bar_kvf + 8 * slot, (uint32_t)((pos / kRing) & 1));
              if (j == 0) { mbar_wait(bar_oe + 8 * t, ((o_items >> t) & 1) ^ 1); o_items ^= 1u << t; }   // the item before left O
              const uint32_t v_s = sKV + slot * kTile;
              mbar_wait(bar_p + 8 * t, ph);
              tcgen05_fence_after();
#pragma unroll
              for (int h = 0; h < 2; ++h)
                mma_ts4<16, 128>(tmem_O + t * HD, tmem_S + t * BN + h * 32, make_smem_desc(v_s + h * 8192, kHalf, 1024), idesc_o, (j | h) ? 1u : 0u);
              if (p.split || t == 1 || j >= it.n1) tcgen05_commit_e(bar_kve + 8 * slot);
              if (j == nt - 1) tcgen05_commit_e(bar_of + 8 * t);
            }
            if (j + 1 < nt) {                      // S over P of this step: behind its PV in pipe order
              issue_s(t, pos0 + at(t, j + 1), false, j + 2 == nt, p.split || t == 1 || j + 1 >= it.n1);
            } else if (j == (nt ? nt : steps_n) - 1) {                  // first S of the next item: this stream's last PV has been issued
              if (!asked) { nx = get(il + 1); asked = true; }
              const int nn = t ? nx.n1 : nx.n0;
              if (nn > 0) issue_s(t, pos1 + at(t, 0), true, nn == 1, p.split || t == 1 || nx.n1 == 0);
            }
          }
        }
        it = nx;
        pos0 = pos1;
      }
    }
    __syncwarp();
  } else if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    const int quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t tO = tmem_O + ((uint32_t)(quarter * 32) << 16), stage = sO + quarter * kStage;
    uint32_t ph = 0;                               // bit t: parity of stream t's items
    for (int il = 0;; ++il) {
      const int idx = item_index(il, true);
      if (idx < 0) break;
      const FwdItem it = fwd_item(idx, p);
      const bool merge = p.split && it.n1 > 0;     // both streams' sums belong to one query tile
#pragma unroll 1
      for (int t = 0; t < (p.split ? 1 : 2); ++t) {
        if ((t ? it.n1 : it.n0) == 0) continue;
        mbar_wait(bar_of + 8 * t, (ph >> t) & 1);
        mbar_wait(bar_lf + 8 * t, (ph >> t) & 1);
        float m, l, f0 = 1.f, f1 = 0.f;
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(m), "=f"(l) : "r"(sStat + t * 1024 + row * 8) : "memory");
        if (merge) {
          mbar_wait(bar_of + 8, 0);
          mbar_wait(bar_lf + 8, 0);
          float m1, l1;
          asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(m1), "=f"(l1) : "r"(sStat + 1024 + row * 8) : "memory");
          const float mm = fmaxf(m, m1);
          f0 = ex2((m - mm) * p.scale_log2);
          f1 = m1 == -INFINITY ? 0.f : ex2((m1 - mm) * p.scale_log2);
          l = l * f0 + l1 * f1;
          m = mm;
        }
        ph ^= 1u << t;
        mbar_arrive(bar_le + 8 * t);
        tcgen05_fence_after();
        const float inv_l = 1.f / l;
        const int r0 = (it.qt + t) * BM + quarter * 32;
        // The rows leave through the warp's stage, 64 columns at a time, so that a store writes four runs of 128 bytes; stored as they come
        // out of TMEM they were 32 runs of 16 bytes an instruction.
        __nv_bfloat16* orow = out + (long)it.b * p.o_sb + (long)(r0 + (lane >> 3)) * p.o_ss + (long)it.head * p.o_sh + (lane & 7) * 8;
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          __syncwarp();                            // what was in the stage has been read
#pragma unroll
          for (int c = 0; c < 4; ++c) {            // 16 columns
            uint32_t r[16];
            tcgen05_ld_32x16(tO + t * HD + h * 64 + c * 16, r);
            if (merge) {
              uint32_t r1[16];
              tcgen05_ld_32x16(tO + HD + h * 64 + c * 16, r1);
              tcgen05_wait_ld();
#pragma unroll
              for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(fmaf(__uint_as_float(r[i]), f0, __uint_as_float(r1[i]) * f1));
            } else {
              tcgen05_wait_ld();
            }
#pragma unroll
            for (int v4 = 0; v4 < 2; ++v4) {
              uint32_t o[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) o[i] = pack_bf16(__uint_as_float(r[v4 * 8 + 2 * i]) * inv_l, __uint_as_float(r[v4 * 8 + 2 * i + 1]) * inv_l);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage + lane * 128 + (((c * 2 + v4) ^ (lane & 7)) * 16)), "r"(o[0]),
                           "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
            }
          }
          if (h == 1) { tcgen05_fence_before(); mbar_arrive(bar_oe + 8 * t); }      // the next item's first product may overwrite O
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {            // rows 4 i + lane / 8
            const int rr = 4 * i + (lane >> 3);
            uint4 o;
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(o.x), "=r"(o.y), "=r"(o.z), "=r"(o.w)
                         : "r"(stage + rr * 128 + (((lane & 7) ^ (rr & 7)) * 16)) : "memory");
            if (r0 + rr < p.S_q) *reinterpret_cast<uint4*>(orow + (long)(4 * i) * p.o_ss + h * 64) = o;
          }
        }
        if (r0 + lane < p.S_q) p.lse[((long)it.b * p.H + it.head) * p.S_q + r0 + lane] = m * p.scale + __logf(l);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
    const int t = warp >= 4;                       // stream of this warpgroup
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t tS = tmem_S + t * BN + lane_base, tO = tmem_O + t * HD + lane_base;
    const uint32_t my_s = bar_s + 8 * t, my_p = bar_p + 8 * t;
    const float sl2 = p.scale_log2;
    const uint64_t sl2_2 = pack2(sl2, sl2);
    int g = 0, items = 0;
    for (int il = 0;; ++il) {
      const int idx = item_index(il, true);
      if (idx < 0) break;
      const FwdItem it = fwd_item(idx, p);
      const int nt = t ? it.n1 : it.n0;
      if (nt == 0) continue;
      const int q0 = (it.qt + (p.split ? 0 : t)) * BM, q_idx = q0 + row;
      float m_ref = -INFINITY, l = 0.f;
      for (int j = 0; j < nt; ++j, ++g) {
        mbar_wait(my_s, (uint32_t)(g & 1));
        tcgen05_fence_after();
        const int kv0 = (p.split ? 2 * j + t : j) * BN;
        const bool masked = (p.causal && kv0 + BN - 1 > q0) || (kv0 + BN > p.S_kv);
        // last visible column of this row, and of the warp's first: most quarters of a tile need no look at single columns
        const int kv_last = p.S_kv - 1 - kv0, lim = p.causal ? min(kv_last, q_idx - kv0) : kv_last;
        const int lim_lo = p.causal ? min(kv_last, q0 + quarter * 32 - kv0) : kv_last;
        // ---- the whole S row (128 fp32) comes into registers with four back-to-back TMEM loads and one wait
        uint32_t sr[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tcgen05_ld_32x32(tS + c * 32, sr[c]);
        tcgen05_wait_ld();
        if (masked) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (lim_lo < c * 32 + 31) fwd_mask(sr[c], lim - c * 32);
        }
        if (j == 0) {
          float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int i = 0; i < 32; i += 2)
#pragma unroll
            for (int c = 0; c < 4; ++c) m4[c] = max3(m4[c], __uint_as_float(sr[c][i]), __uint_as_float(sr[c][i + 1]));
          m_ref = fmaxf(max3(m4[0], m4[1], m4[2]), m4[3]);
        }
        uint64_t shift = pack2(-m_ref * sl2, -m_ref * sl2), sum[4] = {0ull, 0ull, 0ull, 0ull};
        float mx, none;
        fwd_exps<true>(sr, 0, sl2_2, shift, sum[0], mx);
        const bool need = (mx - m_ref) * sl2 > 8.f;
        if (__any_sync(0xffffffffu, need)) {
          const float f = need ? ex2((m_ref - mx) * sl2) : 1.f;
          if (need) m_ref = mx;
          l *= f;
          shift = pack2(-m_ref * sl2, -m_ref * sl2);
          if (j > 0) {                             // PV of the step before is done (this S came after it): O is quiescent
#pragma unroll 1
            for (int c = 0; c < 8; ++c) {
              uint32_t r[16];
              tcgen05_ld_32x16(tO + c * 16, r);
              tcgen05_wait_ld();
#pragma unroll
              for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * f);
              tcgen05_st_32x16(tO + c * 16, r);
            }
          }
          tcgen05_ld_32x32(tS, sr[0]);
          tcgen05_wait_ld();
          if (masked) fwd_mask(sr[0], lim);
          sum[0] = 0ull;
          fwd_exps<false>(sr, 0, sl2_2, shift, sum[0], none);
        }
        if (!(mx < INFINITY)) l = __int_as_float(0x7fffffff);        // NaN or +inf among the scores: a row of NaN
        tcgen05_st_32x16p(tS, sr[0]);
#pragma unroll
        for (int c = 1; c < 4; ++c) {
          fwd_exps<false>(sr, c, sl2_2, shift, sum[c], none);
          tcgen05_st_32x16p(tS + c * 16, sr[c]);
        }
        tcgen05_wait_st();
        tcgen05_fence_before();
        mbar_arrive(my_p);
        float l4[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) { float a, b; unpack2(sum[c], a, b); l4[c] = a + b; }
        l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
      }
      // ---- maximum and row sum to the output warps
      mbar_wait(bar_le + 8 * t, (uint32_t)((items & 1) ^ 1));
      ++items;
      asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(sStat + t * 1024 + row * 8), "f"(m_ref), "f"(l) : "memory");
      mbar_arrive(bar_lf + 8 * t);
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 13) tcgen05_dealloc(tmem_base, 512);
}

// ====================================================================================================================
// Backward.  One CTA per (128-row KV tile, kv head or a part of its query heads, batch); it keeps K/V resident in smem and dK/dV
// resident in TMEM and walks the 64-row query tiles (× the query heads of its part) that can see this KV tile.  Everything is computed transposed so that the
// softmax threads own a *kv* row and P/dS land directly in the operand layouts the next GEMMs need:
//   Sᵀ  = K·Qᵀ        (A = K  K-major, B = Q  K-major)            → TMEM [128 kv × 64 q]
//   dPᵀ = V·dOᵀ       (A = V  K-major, B = dO K-major)            → TMEM [128 kv × 64 q]
//   Pᵀ = exp2(Sᵀ·c − lse₂[q]) ;  dSᵀ = Pᵀ ∘ (dPᵀ·scale − δ[q]·scale)   (thread = kv row; lse₂/δ broadcast from smem)
//   dV += Pᵀ·dO       (A = Pᵀ from TMEM (in place over Sᵀ), B = dO MN-major)
//   dK += dSᵀ·Q       (A = dSᵀ from TMEM (over dPᵀ),       B = Q  MN-major)
//   dQᵀ = Kᵀ·dSᵀ      (A = K MN-major, B = dSᵀ MN-major)          → TMEM [128 d × 64 q], drained by a second warpgroup
//                      into smem and added to the fp32 dQ accumulator with one bulk async reduce (no per-element atomics).
// warp 0 TMA, warp 1 MMA issue, warps 2-5 and 6-9 softmax/dS of the first and last 32 query columns (+ dK / dV epilogue), warps 10-13 dQ drain.
// A step of one query tile takes about 1850 cycles: its products 1660 (1280 of mathematics; operands of 64 columns are read from shared memory
// faster than they are used), the softmax chain of a step about as long.  One softmax warpgroup (64 exponentials a thread) made it 2070, and
// one 16 KB stage for the sums of dQ, which the drain waited for, 2250.  Start and end of a block are 10 thousand cycles more, two thirds of
// them the stores of dK and dV at 32 bytes a cycle and SM beside the last sums of dQ.  Main kernel, 1 x 2048 tokens, 32 heads: 116 us then, 88 now.
constexpr int BQ = 64;
constexpr int kThreadsBwd = 448;
constexpr int kQStages = 3;
constexpr uint32_t kQTile = BQ * HD * 2;                        // 16 KB
constexpr uint32_t kOffK = 0, kOffV = kTile, kOffQ = 2 * kTile, kOffdO = kOffQ + kQStages * kQTile,
                   kOffdS = kOffdO + kQStages * kQTile, kOffdQ = kOffdS + 2 * kQTile, kOffStats = kOffdQ + 2 * 16384,
                   kOffBars = kOffStats + kQStages * 512;
constexpr uint32_t kSmemBwd = kOffBars + 256 + 1024;

struct BwdParams {
  int S_q, S_kv, H, Hkv, B, S_pad;
  Coord q, k, v, g;
  long dk_sb, dk_ss, dk_sh, dv_sb, dv_ss, dv_sh;
  float scale, scale_log2;
  int causal;
  int group_bh;                // (batch, KV head, part) triples whose Q / dO / dQ stay in L2 together
  int parts;                   // blocks that share the query heads of one KV head (divides the group)
  float* kv_part;              // parts > 1: fp32 dK and dV of each part, [2][B, Hkv, parts][S_kv, 128]
  const float* stats;          // [2][B*H*S_pad (+pad)] : −lse·log2e , −δ·scale
  long stats_stride;
  float* dq_acc;               // [B, H, S_pad, 128] fp32
  unsigned* turnstile;         // DET only: [B, H, ceil(S_q / BQ)] contributions already added to each dQ tile
};

NXD_DEVICE void bulk_load_1d(uint32_t smem_dst, const void* gsrc, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_dst), "l"(gsrc), "r"(bytes), "r"(bar) : "memory");
}
NXD_DEVICE void bulk_reduce_add_f32(void* gdst, uint32_t smem_src, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;"
               ::"l"(gdst), "r"(smem_src), "r"(bytes) : "memory");
}
NXD_DEVICE void named_bar(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

// Softmax-side math of one backward tile, split in two phases so the exp work (needs only Sᵀ, which the tensor pipe delivered a
// full iteration ago) runs while dPᵀ of the same tile is still being computed:
//   phase 1: Pᵀ = exp2(Sᵀ·c − lse₂[q])  → fp32 in registers (pf) + bf16 pairs packed in place into sv (element pair (i,i+1) → i/2)
//   phase 2: dSᵀ = Pᵀ ∘ (dPᵀ·scale − δ[q]·scale) → bf16 pairs packed in place into dpv
// The stats rows hold −lse·log2e and −δ·scale so both affine steps are single packed FMAs; MASKED is a template parameter so
// the common tile has no per-element branches or selects.
template <bool MASKED>
NXD_DEVICE void bwd_p_math(uint32_t (&sv)[32], float (&pf)[32], uint32_t stats_s, float sl2, int kv, int q0, int S_q, int S_kv, int causal) {
  const uint64_t sl2_2 = pack2(sl2, sl2);
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    float4 l2;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(l2.x), "=f"(l2.y), "=f"(l2.z), "=f"(l2.w) : "r"(stats_s + i * 4));
    const uint64_t nl2[2] = {pack2(l2.x, l2.y), pack2(l2.z, l2.w)};
#pragma unroll
    for (int e2 = 0; e2 < 2; ++e2) {
      float x0, x1;
      unpack2(fma2(pack2u(sv[i + 2 * e2], sv[i + 2 * e2 + 1]), sl2_2, nl2[e2]), x0, x1);
      float p0 = ex2(x0), p1 = ex2(x1);
      if constexpr (MASKED) {
        const int q = q0 + i + 2 * e2;
        p0 = (kv < S_kv && q < S_q && (!causal || kv <= q)) ? p0 : 0.f;          // selects; also kills NaN padding
        p1 = (kv < S_kv && q + 1 < S_q && (!causal || kv <= q + 1)) ? p1 : 0.f;
      }
      pf[i + 2 * e2] = p0;
      pf[i + 2 * e2 + 1] = p1;
    }
    sv[i >> 1] = pack_bf16(pf[i], pf[i + 1]);
    sv[(i >> 1) + 1] = pack_bf16(pf[i + 2], pf[i + 3]);
  }
}

template <bool MASKED>
NXD_DEVICE void bwd_ds_math(uint32_t (&dpv)[32], const float (&pf)[32], uint32_t stats_s, float sc) {
  const uint64_t sc_2 = pack2(sc, sc);
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    float4 dl;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(dl.x), "=f"(dl.y), "=f"(dl.z), "=f"(dl.w) : "r"(stats_s + 256 + i * 4));
    const uint64_t ndl[2] = {pack2(dl.x, dl.y), pack2(dl.z, dl.w)};
    float dsv[4];
#pragma unroll
    for (int e2 = 0; e2 < 2; ++e2) {
      float d0, d1;
      unpack2(mul2(pack2(pf[i + 2 * e2], pf[i + 2 * e2 + 1]), fma2(pack2u(dpv[i + 2 * e2], dpv[i + 2 * e2 + 1]), sc_2, ndl[e2])), d0, d1);
      if constexpr (MASKED) {            // P is already exactly 0 where masked, but 0·NaN (padding garbage) must not leak
        d0 = pf[i + 2 * e2] == 0.f ? 0.f : d0;
        d1 = pf[i + 2 * e2 + 1] == 0.f ? 0.f : d1;
      }
      dsv[2 * e2] = d0; dsv[2 * e2 + 1] = d1;
    }
    dpv[i >> 1] = pack_bf16(dsv[0], dsv[1]);
    dpv[(i >> 1) + 1] = pack_bf16(dsv[2], dsv[3]);
  }
}

// DET = deterministic dQ: the contributions of the K/V tiles to one dQ tile are added in K/V-tile order through a turnstile
// counter per (batch, head, query tile) — CTA n of a (batch, KV head) column waits until n earlier tiles have landed, adds its
// own with the same bulk reduce, waits for that reduce to COMPLETE and releases the next.  CTAs are dispatched in increasing
// blockIdx.x, in which a column's tiles ascend, so the CTA being waited for is always resident or done.  Slower (the drain of a tile is serialised across the
// column), bit-reproducible.  DET = false compiles to exactly the kernel without the option.
template <bool DET>
__global__ void __launch_bounds__(kThreadsBwd, 1)
fa_bwd_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
              const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tg,
              __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv, const BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sK = base + kOffK, sV = base + kOffV, sQ = base + kOffQ, sdO = base + kOffdO, sdS = base + kOffdS,
                 sdQ = base + kOffdQ, sStats = base + kOffStats, bars = base + kOffBars;
  // barriers: k | qf[3] | qe[3] | s[2] | dp | p | dq | dqr | acc | v | tmem slot
  const uint32_t bar_k = bars, bar_v = bars + 112, bar_qf = bars + 8, bar_qe = bars + 32, bar_s = bars + 56, bar_dp = bars + 72,
                 bar_p = bars + 80, bar_dq = bars + 88, bar_dqr = bars + 96, bar_acc = bars + 104, tmem_slot = bars + 128;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Blocks start heaviest first (causal: the first K/V tiles see the most query tiles) within groups of heads that share L2: head by
  // head, the last heads' heavy tiles started when most SMs had nothing left (1 x 2048 x 32 heads: 142 us, now 119).
  int n, kvh, b, vh;                                       // vh: the part's index among all parts of all KV heads
  const int heads_v = p.Hkv * p.parts;
  {
    const int tiles = (p.S_kv + BN - 1) / BN, bhs = p.B * heads_v;
    const int grp = (int)blockIdx.x / (tiles * p.group_bh), rem = (int)blockIdx.x - grp * tiles * p.group_bh;
    const int gs = min(p.group_bh, bhs - grp * p.group_bh), bh = grp * p.group_bh + rem % gs;
    n = rem / gs;
    vh = bh % heads_v;
    kvh = vh / p.parts;
    b = bh / heads_v;
  }
  const int group = p.H / heads_v;                         // query heads of this block: vh * group ...
  const int nq = (p.S_q + BQ - 1) / BQ;
  const int t0 = p.causal ? (n * BN) / BQ : 0;
  const int per_head = nq - t0;
  const int n_iter = per_head * group;
  const int kv0 = n * BN;

  if (threadIdx.x == 0) {
    mbar_init(bar_k, 1); mbar_init(bar_v, 1);
    for (int i = 0; i < kQStages; ++i) { mbar_init(bar_qf + 8 * i, 1); mbar_init(bar_qe + 8 * i, 1); }
    mbar_init(bar_s, 1); mbar_init(bar_s + 8, 1);
    mbar_init(bar_dp, 1); mbar_init(bar_p, 256); mbar_init(bar_dq, 1); mbar_init(bar_dqr, 128);
    mbar_init(bar_acc, 1);
    fence_barrier_init();
    // K, V and the first tile of Q and dO are on their way while the tensor memory is allocated; what the kernel before this one writes (the
    // statistics) is not among them
    if (n_iter > 0) {
      const int kh = kvh * p.k.h, kb = b * p.k.b, v_h = kvh * p.v.h, vb = b * p.v.b, head = vh * group;
      mbar_expect_tx(bar_k, kTile);
      tma_load_4d(sK, &tk, bar_k, 0, kv0, kh, kb);
      tma_load_4d(sK + kHalf, &tk, bar_k, 64, kv0, kh, kb);
      mbar_expect_tx(bar_qf, 2 * kQTile + 512);
      tma_load_4d(sQ, &tq, bar_qf, 0, t0 * BQ, head * p.q.h, b * p.q.b);
      tma_load_4d(sQ + kQTile / 2, &tq, bar_qf, 64, t0 * BQ, head * p.q.h, b * p.q.b);
      mbar_expect_tx(bar_v, kTile);
      tma_load_4d(sV, &tv, bar_v, 0, kv0, v_h, vb);
      tma_load_4d(sV + kHalf, &tv, bar_v, 64, kv0, v_h, vb);
      tma_load_4d(sdO, &tg, bar_qf, 0, t0 * BQ, head * p.g.h, b * p.g.b);
      tma_load_4d(sdO + kQTile / 2, &tg, bar_qf, 64, t0 * BQ, head * p.g.h, b * p.g.b);
    }
  }
  if (warp == 1) {
    tcgen05_alloc(tmem_slot, 512);
    tcgen05_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  pdl_trigger();                                           // fa_bwd_dq_out_kernel's blocks wait on the SMs that run out of this kernel's
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  // TMEM columns: dK [0,128) | dV [128,256) | Sᵀ/Pᵀ double buffer [256,384) | dPᵀ [384,448) | dQᵀ [448,512)
  const uint32_t tmem_dK = tmem_base, tmem_dV = tmem_base + 128, tmem_ST = tmem_base + 256, tmem_dP = tmem_base + 384,
                 tmem_dQ = tmem_base + 448;

  if (warp == 0) {
    if (lane == 0 && n_iter > 0) {
      pdl_wait();                                          // the statistics come from the kernel before
      for (int it = 0; it < n_iter; ++it) {
        const int qs = it % kQStages;
        const uint32_t ph = (uint32_t)((it / kQStages) & 1);
        const int head = vh * group + it / per_head, t = t0 + it % per_head;
        const uint32_t full = bar_qf + 8 * qs;
        if (it > 0) {
          mbar_wait(bar_qe + 8 * qs, ph ^ 1);
          mbar_expect_tx(full, 2 * kQTile + 512);
          const int qh = head * p.q.h, qb = b * p.q.b, gh = head * p.g.h, gb = b * p.g.b;
          tma_load_4d(sQ + qs * kQTile, &tq, full, 0, t * BQ, qh, qb);
          tma_load_4d(sQ + qs * kQTile + kQTile / 2, &tq, full, 64, t * BQ, qh, qb);
          tma_load_4d(sdO + qs * kQTile, &tg, full, 0, t * BQ, gh, gb);
          tma_load_4d(sdO + qs * kQTile + kQTile / 2, &tg, full, 64, t * BQ, gh, gb);
        }
        const float* st = p.stats + ((long)b * p.H + head) * p.S_pad + t * BQ;
        bulk_load_1d(sStats + qs * 512, st, 256, full);
        bulk_load_1d(sStats + qs * 512 + 256, st + p.stats_stride, 256, full);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (n_iter > 0) {   // all 32 lanes run the issue loop; one elected lane executes each tcgen05 instruction
      constexpr uint32_t idesc_s = make_idesc(false, false, 128, BQ);      // Sᵀ, dPᵀ
      constexpr uint32_t idesc_acc = make_idesc(false, true, 128, HD);     // dK, dV
      constexpr uint32_t idesc_dq = make_idesc(true, true, 128, BQ);       // dQᵀ
      mbar_wait(bar_k, 0);
      // Issue order per iteration `it` (everything on the tensor pipe retires in this order):
      //   … Sᵀ_{it+1} already issued …  | wait softmax(it) | dK_it | dPᵀ_{it+1} | dV_it | dQᵀ_it | Sᵀ_{it+2}
      // so while the softmax warps work on tile it+1 the pipe runs dK/dV/dQ of tile it and Sᵀ of tile it+2.
      auto issue_st = [&](int it) {
        const int qs = it % kQStages, st = it & 1;
        mbar_wait(bar_qf + 8 * qs, (uint32_t)((it / kQStages) & 1));
        tcgen05_fence_after();
        const uint32_t q_s = sQ + qs * kQTile;
        mma_ss8<kHalf / 16, 2, kQTile / 32, 2>(tmem_ST + st * BQ, make_smem_desc(sK, 16, 1024), make_smem_desc(q_s, 16, 1024), idesc_s, 0u, bar_s + 8 * st);
      };
      auto issue_dp = [&](int it) {
        const int qs = it % kQStages;
        mbar_wait(bar_qf + 8 * qs, (uint32_t)((it / kQStages) & 1));
        tcgen05_fence_after();
        const uint32_t g_s = sdO + qs * kQTile;
        mma_ss8<kHalf / 16, 2, kQTile / 32, 2>(tmem_dP, make_smem_desc(sV, 16, 1024), make_smem_desc(g_s, 16, 1024), idesc_s, 0u, bar_dp);
      };
      issue_st(0);
      mbar_wait(bar_v, 0);
      issue_dp(0);
      if (n_iter > 1) issue_st(1);
      for (int it = 0; it < n_iter; ++it) {
        const int qs = it % kQStages, st = it & 1;
        mbar_wait(bar_p, (uint32_t)(it & 1));             // Pᵀ_it over Sᵀ_it, dSᵀ_it over dPᵀ_it in TMEM and in smem
        tcgen05_fence_after();
        const uint32_t q_s = sQ + qs * kQTile, g_s = sdO + qs * kQTile, ds_s = sdS + st * kQTile;
        mma_ts4<32, 128>(tmem_dK, tmem_dP, make_smem_desc(q_s, kQTile / 2, 1024), idesc_acc, it ? 1u : 0u);
        if (it + 1 < n_iter) issue_dp(it + 1);            // over dSᵀ_it: behind dK_it in pipe order
        mma_ts4<32, 128>(tmem_dV, tmem_ST + st * BQ, make_smem_desc(g_s, kQTile / 2, 1024), idesc_acc, it ? 1u : 0u);
        tcgen05_commit_e(bar_qe + 8 * qs);
        if (it >= 1) {
          mbar_wait(bar_dqr, (uint32_t)((it - 1) & 1));   // dQᵀ_{it-1} has been read out of TMEM
          tcgen05_fence_after();
        }
        mma_ss8<512, 128, 512, 128>(tmem_dQ, make_smem_desc(sK, kHalf, 1024), make_smem_desc(ds_s, kHalf, 1024), idesc_dq, 0u, bar_dq);
        if (it + 2 < n_iter) issue_st(it + 2);            // overwrites Pᵀ_it — after dV_it in pipe order
      }
      tcgen05_commit_e(bar_acc);
    }
    __syncwarp();
  } else if (warp < 10) {
    // ===== softmax / dS warps: thread = kv row, 32 of the tile's query columns =====
    const int quarter = warp & 3, wg = (warp - 2) >> 2;
    const int row = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const int kv = kv0 + row;
    const float sl2 = p.scale_log2, sc = p.scale;
    int qs = 0, t = t0;
    uint32_t ph = 0;
    for (int it = 0; it < n_iter; ++it) {
      const int st = it & 1;
      const int q0 = t * BQ;
      const uint32_t tS = tmem_ST + st * BQ + wg * 32 + lane_base, tdP = tmem_dP + wg * 32 + lane_base;
      mbar_wait(bar_qf + 8 * qs, ph);                                  // stats (TMA-written) visible to this thread
      mbar_wait(bar_s + 8 * st, (uint32_t)((it >> 1) & 1));
      tcgen05_fence_after();
      const bool masked = (p.causal && q0 < kv0 + BN - 1) || (q0 + BQ > p.S_q) || (kv0 + BN > p.S_kv);
      const uint32_t stats_s = sStats + qs * 512 + wg * 128;
      const uint32_t ds_row = sdS + st * kQTile + row * 128;
      // ---- phase 1 (needs only Sᵀ): Pᵀ, written back over Sᵀ in TMEM (each half over its own columns)
      uint32_t sv[32];
      float pf[32];
      tcgen05_ld_32x32(tS, sv);
      tcgen05_wait_ld();
      if (masked) bwd_p_math<true>(sv, pf, stats_s, sl2, kv, q0 + wg * 32, p.S_q, p.S_kv, p.causal);
      else bwd_p_math<false>(sv, pf, stats_s, sl2, kv, q0 + wg * 32, p.S_q, p.S_kv, p.causal);
      tcgen05_st_32x16p(tS, sv);
      // ---- phase 2 (dPᵀ of this tile was issued while phase 1 ran): dSᵀ → TMEM and smem
      mbar_wait(bar_dp, (uint32_t)(it & 1));
      tcgen05_fence_after();
      uint32_t dpv[32];
      tcgen05_ld_32x32(tdP, dpv);
      tcgen05_wait_ld();
      if (masked) bwd_ds_math<true>(dpv, pf, stats_s, sc);
      else bwd_ds_math<false>(dpv, pf, stats_s, sc);
      tcgen05_st_32x16p(tdP, dpv);
      // dSᵀ row → smem, 128B-swizzled: 16-byte chunk c of row r lives at chunk (c ^ (r & 7))
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint32_t chunk = (uint32_t)(wg * 4 + c) ^ (uint32_t)(row & 7);
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(ds_row + chunk * 16), "r"(dpv[c * 4]),
                     "r"(dpv[c * 4 + 1]), "r"(dpv[c * 4 + 2]), "r"(dpv[c * 4 + 3]) : "memory");
      }
      tcgen05_wait_st();
      fence_async_smem();
      tcgen05_fence_before();
      mbar_arrive(bar_p);
      if (++qs == kQStages) { qs = 0; ph ^= 1; }
      if (++t == nq) t = t0;
    }
    // ---- epilogue: dK by the first warpgroup, dV by the second, through the shared memory of K .. dO, which nothing reads any more (bar_acc:
    //      every product is done), so that a store writes whole rows.  In small loops: unrolled, most of its time went into fetching
    //      instructions that run once a block.
    if (n_iter > 0) {
      mbar_wait(bar_acc, 0);
      tcgen05_fence_after();
    }
    // 16-byte chunk c of the warp's row i stands at chunk c ^ (i & 7); rows of 256 bytes of bf16 (a store: two rows) or 512 of fp32 (one)
    const bool f32 = p.parts > 1;
    const uint32_t acc = (wg ? tmem_dV : tmem_dK) + lane_base, pitch = f32 ? 512 : 256;
    const uint32_t stage = sK + wg * 2 * kTile + quarter * 32 * pitch, mine = stage + lane * pitch;
    const int r0 = kv0 + quarter * 32;
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {                          // 32 columns
      uint32_t r[32];
      if (n_iter > 0) {
        tcgen05_ld_32x32(acc + c * 32, r);
        tcgen05_wait_ld();
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) r[i] = 0;
      }
      if (f32) {
#pragma unroll
        for (int v4 = 0; v4 < 8; ++v4)
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(mine + (((c * 8 + v4) ^ (lane & 7)) * 16)), "r"(r[v4 * 4]), "r"(r[v4 * 4 + 1]),
                       "r"(r[v4 * 4 + 2]), "r"(r[v4 * 4 + 3]) : "memory");
      } else {
#pragma unroll
        for (int v4 = 0; v4 < 4; ++v4) {
          uint32_t o[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) o[i] = pack_bf16(__uint_as_float(r[v4 * 8 + 2 * i]), __uint_as_float(r[v4 * 8 + 2 * i + 1]));
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(mine + (((c * 4 + v4) ^ (lane & 7)) * 16)), "r"(o[0]), "r"(o[1]), "r"(o[2]),
                       "r"(o[3]) : "memory");
        }
      }
    }
    __syncwarp();
    const int chunks = f32 ? 32 : 16, c = lane & (chunks - 1), step = 32 / chunks;
    const long row_bytes = f32 ? HD * 4 : (wg ? p.dv_ss : p.dk_ss) * 2;
    char* dst = f32 ? (char*)(p.kv_part + ((((long)wg * p.B + b) * heads_v + vh) * p.S_kv + r0) * HD)
                    : (char*)((wg ? dv + (long)b * p.dv_sb + (long)kvh * p.dv_sh : dk + (long)b * p.dk_sb + (long)kvh * p.dk_sh) + (long)r0 * (row_bytes / 2));
#pragma unroll 4
    for (int i = lane / chunks; i < 32; i += step) {
      uint4 o;
      asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(o.x), "=r"(o.y), "=r"(o.z), "=r"(o.w)
                   : "r"(stage + i * pitch + ((c ^ (i & 7)) * 16)) : "memory");
      if (r0 + i < p.S_kv) *reinterpret_cast<uint4*>(dst + i * row_bytes + c * 16) = o;
    }
  } else {
    // ===== dQ drain warps: thread = head-dim index d (TMEM lane), columns = q =====
    const int quarter = warp & 3;
    const int d = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const int tid = threadIdx.x - 320;
    if (tid == 0) pdl_wait();                              // which zeroes what is added to here
    for (int it = 0; it < n_iter; ++it) {
      const int st = it & 1;
      const int head = vh * group + it / per_head, t = t0 + it % per_head;
      mbar_wait(bar_dq, (uint32_t)(it & 1));
      tcgen05_fence_after();
      float* gdst = p.dq_acc + (((long)b * p.H + head) * p.S_pad + (long)t * BQ) * HD;
      uint32_t r[2][32];
      tcgen05_ld_32x32(tmem_dQ + lane_base, r[0]);
      tcgen05_ld_32x32(tmem_dQ + lane_base + 32, r[1]);
      tcgen05_wait_ld();
      tcgen05_fence_before();
      mbar_arrive(bar_dqr);                     // the MMA warp may overwrite dQᵀ with the next tile right away
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (tid == 0) bulk_wait_read1();        // the bulk reduce before the last has finished reading its half of the stage
        named_bar(1, 128);
#pragma unroll
        for (int c = 0; c < 32; ++c)
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(sdQ + h * 16384 + c * 512 + d * 4), "r"(r[h][c]) : "memory");
        fence_async_smem();
        named_bar(1, 128);
        if (tid == 0) {
          if constexpr (DET) {
            if (h == 0) {                           // my turn: the n earlier K/V tiles of this column have been added
              const unsigned* turn = p.turnstile + ((long)b * p.H + head) * nq + t;
              unsigned seen, spins = 0;
              unsigned long long t_start = 0;
              do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(turn) : "memory");
                if (seen < (unsigned)n && (++spins & 0x3ffu) == 0) {
                  unsigned long long now;
                  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
                  if (t_start == 0) t_start = now;
                  else if (now - t_start > 10000000000ull) __trap();          // an earlier tile never arrived
                }
              } while (seen < (unsigned)n);
            }
          }
          bulk_reduce_add_f32(gdst + (long)h * 32 * HD, sdQ + h * 16384, 16384);
          bulk_commit();
          if constexpr (DET) {
            if (h == 1) {                           // both halves of the tile are in memory before the next CTA may add
              bulk_wait0();
              __threadfence();
              unsigned* turn = p.turnstile + ((long)b * p.H + head) * nq + t;
              asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(turn), "r"(1u) : "memory");
            }
          }
        }
      }
    }
    if (tid == 0) bulk_wait0();
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) tcgen05_dealloc(tmem_base, 512);
}

// −δ·scale and −lse·log2e per (b, h, s), and zeros for the row's dQ accumulator (rows up to S_pad).  16 lanes per row, 16 bytes per
// lane; heads fastest, as o and dO lie in memory.  The main kernel's blocks take their places and load K, V, Q and dO beside this one, and the
// conversion of dQ starts on the SMs that run out of it: whole backward with a main kernel of 116 us, 1 x 2048 x 32 heads, 146 us with launches
// one after the other, 140 so, 136 with one row per half warp instead of four in flight; 1 x 1000 x 32: 61 and 53; 1 x 70 x 32: 21.6 and 14.5.
__global__ void __launch_bounds__(256) fa_bwd_prep_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ go,
                                   const float* __restrict__ lse, const float* __restrict__ dlse, float* __restrict__ stats,
                                   float* __restrict__ dq_acc, long stats_stride, int B, int S,
                                   int H, int S_pad, long o_sb, long o_ss, long o_sh, long g_sb, long g_ss, long g_sh,
                                   float scale) {
  pdl_trigger();
  const int lane = threadIdx.x & 15, bh = B * H;
  const long r = (long)blockIdx.x * 16 + (threadIdx.x >> 4);
  const int s = r < (long)S_pad * bh ? (int)(r / bh) : S_pad, in = (int)(r % bh), h = in % H, b = in / H;
  Pack16<__nv_bfloat16> ov, gv;
  if (s < S) {
    ov.load_nc(o + b * o_sb + s * o_ss + h * o_sh + lane * 8);
    gv.load_nc(go + b * g_sb + s * g_ss + h * g_sh + lane * 8);
  }
  if (s < S_pad) {
    float4* z = reinterpret_cast<float4*>(dq_acc + (((long)b * H + h) * S_pad + s) * HD) + lane;
    z[0] = z[16] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float acc = 0.f;
  if (s < S) {
#pragma unroll
    for (int j = 0; j < 8; ++j) acc += ov.f(j) * gv.f(j);
  }
#pragma unroll
  for (int m = 8; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
  if (lane == 0 && s < S) {
    const long row = (long)b * H + h, idx = row * S_pad + s;
    stats[idx] = -lse[row * S + s] * 1.4426950408889634f;
    // a gradient flowing into LSE itself (ring attention merges blocks through their LSEs) adds g_lse·P to dS, i.e. it
    // simply shifts δ: dS = P∘(dP − (δ − g_lse))
    const float g_lse = dlse ? dlse[row * S + s] : 0.f;
    stats[stats_stride + idx] = -(acc - g_lse) * scale;
  }
}

// fp32 dQ accumulator [B,H,S_pad,128] → bf16 dq with arbitrary (b, s, h) strides; 8 elements per thread.
__global__ void fa_bwd_dq_out_kernel(const float* acc, __nv_bfloat16* dq, int B, int S, int H,
                                     int S_pad, long sb, long ss, long sh) {
  pdl_trigger();
  pdl_wait();
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;        // over B*H*S*16
  if (i >= (long)B * H * S * 16) return;
  const int c = (int)(i & 15);
  const long r = i >> 4;
  const int s = (int)(r % S), h = (int)((r / S) % H), b = (int)(r / ((long)S * H));
  const float4* src = reinterpret_cast<const float4*>(acc + (((long)b * H + h) * S_pad + s) * HD + c * 8);
  const float4 x = src[0], y = src[1];
  uint4 o;
  o.x = pack_bf16(x.x, x.y); o.y = pack_bf16(x.z, x.w); o.z = pack_bf16(y.x, y.y); o.w = pack_bf16(y.z, y.w);
  *reinterpret_cast<uint4*>(dq + b * sb + s * ss + h * sh + c * 8) = o;
}

// dK and dV of a KV head out of the fp32 sums of its parts, added in their order; 8 elements per thread.
__global__ void fa_bwd_kv_out_kernel(const float* part, __nv_bfloat16* dk, __nv_bfloat16* dv, int B,
                                     int S, int Hkv, int parts, long k_sb, long k_ss, long k_sh, long v_sb, long v_ss, long v_sh) {
  pdl_wait();
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x, n = (long)B * Hkv * S * 16;        // over 2 * B*Hkv*S*16
  if (i >= 2 * n) return;
  const bool is_v = i >= n;
  const int c = (int)(i & 15);
  const long r = (is_v ? i - n : i) >> 4;
  const int s = (int)(r % S), h = (int)((r / S) % Hkv), b = (int)(r / ((long)S * Hkv));
  const float* src = part + (((((long)is_v * B + b) * Hkv + h) * parts) * S + s) * HD + c * 8;
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
  for (int j = 0; j < parts; ++j) {
    const float4 a = reinterpret_cast<const float4*>(src + (long)j * S * HD)[0], e = reinterpret_cast<const float4*>(src + (long)j * S * HD)[1];
    x.x += a.x; x.y += a.y; x.z += a.z; x.w += a.w;
    y.x += e.x; y.y += e.y; y.z += e.z; y.w += e.w;
  }
  uint4 o;
  o.x = pack_bf16(x.x, x.y); o.y = pack_bf16(x.z, x.w); o.z = pack_bf16(y.x, y.y); o.w = pack_bf16(y.z, y.w);
  __nv_bfloat16* dst = is_v ? dv + b * v_sb + s * v_ss + h * v_sh : dk + b * k_sb + s * k_ss + h * k_sh;
  *reinterpret_cast<uint4*>(dst + c * 8) = o;
}

// ---- host side -----------------------------------------------------------------------------------------------------
// A [B, S, H, 128] bf16 view with strides (sb, ss, sh, 1) as a map of four dimensions, so that rows behind the S-th of a (batch, head) read
// as zeros: masked keys have probability 0, and 0 x NaN of whatever lies there (another sequence, a cache's old rows) would be NaN.
struct View { const void* ptr; int B, S, H; long sb, ss, sh; };

static CUtensorMap view_tmap(const View& v, Coord& c, uint32_t box_rows = 128) {
  // strides as the callers prepare them (ops/attention.py _tma_view): heads and sequences whole rows apart, or beside one another within a row
  long cols = HD;
  for (const auto& [stride, n] : {std::pair<long, int>{v.sb, v.B}, {v.sh, v.H}})
    if (n > 1 && !(v.ss > 0 && stride >= v.ss && stride % v.ss == 0)) cols += (n - 1) * stride;
  if (cols > v.ss && v.S > 1) nxd_throw("attention: unsupported q/k/v strides", __FILE__, __LINE__);
  c = Coord{v.H > 1 && v.sh != 0, v.B > 1 && v.sb != 0};
  const long ss = v.S > 1 ? v.ss : HD, sh = c.h ? v.sh : HD, sb = c.b ? v.sb : HD;        // of dimensions of one: any
  if ((ss | sh | sb) % 8 || ((uintptr_t)v.ptr % 16)) nxd_throw("attention: q/k/v must be 16-byte aligned", __FILE__, __LINE__);
  return make_tmap_bf16_heads(v.ptr, {(uint64_t)HD, (uint64_t)v.S, (uint64_t)(c.h ? v.H : 1), (uint64_t)(c.b ? v.B : 1)},
                              {(uint64_t)ss, (uint64_t)sh, (uint64_t)sb}, 64, box_rows);
}

}  // namespace fa

int device_sm_count();

void flash_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse, int B, int S_q, int S_kv, int H,
                    int Hkv, const long* qs, const long* ks, const long* vs, const long* os, float scale, bool causal,
                    cudaStream_t st) {
  using namespace fa;
  if (causal && S_q != S_kv) nxd_throw("attention: causal needs S_q == S_kv", __FILE__, __LINE__);
  if (S_kv <= 0 && (long)S_q * H * B > 0) nxd_throw("attention: no keys", __FILE__, __LINE__);      // the kernel's items have a K / V tile
  FwdParams p;
  p.S_q = S_q; p.S_kv = S_kv; p.H = H; p.Hkv = Hkv; p.B = B;
  const CUtensorMap tq = view_tmap(View{q, B, S_q, H, qs[0], qs[1], qs[2]}, p.q);
  const CUtensorMap tk = view_tmap(View{k, B, S_kv, Hkv, ks[0], ks[1], ks[2]}, p.k);
  const CUtensorMap tv = view_tmap(View{v, B, S_kv, Hkv, vs[0], vs[1], vs[2]}, p.v);
  p.o_sb = os[0]; p.o_ss = os[1]; p.o_sh = os[2];
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.causal = causal ? 1 : 0;
  p.lse = lse;
  NXD_ALLOW_SMEM(fa_fwd_kernel, kSmemFwd);
  const long kv_bytes = (long)S_kv * HD * 4 * Hkv / H;            // K and V of one query head (its share of the group's)
  p.group_bh = (int)std::min<long>((long)H * B, std::max<long>(1, (48l << 20) / std::max<long>(1, kv_bytes)));
  const int sms = device_sm_count();
  const int nq = (S_q + BM - 1) / BM;
  p.split = (long)nq * H * B <= sms;
  const long items = (long)(p.split ? nq : (nq + 1) / 2) * H * B;
  if (items == 0) return;
  // not a dependent: blocks that start early upset the order of the items (1 x 1531 tokens, 64 heads on 8: 57.2 us, 59 as one)
  fa_fwd_kernel<<<(unsigned)items, kThreads, kSmemFwd, st>>>(tq, tk, tv, (__nv_bfloat16*)out, p);
  NXD_CUDA_CHECK(cudaGetLastError());
}

// Blocks per KV head.  Unit: one 64-row query tile, about 1 us.  A launch lasts as long as its heaviest block, or as the sum of all over
// the SMs and, since causal blocks differ, a quarter of the heaviest at the end; equal blocks come in whole rounds.  Every block costs
// six tiles of start and end, every part 256 KB of fp32 sums written and read (0.03 over the chip).  Taken where the estimate falls by a
// twentieth.  The sums are at most twice the fp32 dQ buffer.  Whole backward, caches warm, one block per KV head and by this rule:
//   1 x 2048 tokens, 32 heads on 8: 162 and 113 us;  64 on 8: 310 and 206;  1 x 4096, 32 on 2: 1058 and 351;  64 on 8: 873 and 704;
//   1 x 512, 32 on 8: 57 and 35;  16 on 1: 178 and 33.  Left whole: 1 x 4096, 32 on 8 (342; two parts 357), 2 x 2048 (202; 242).
int flash_attn_bwd_parts(int B, int S_q, int S_kv, int H, int Hkv, bool causal) {
  using namespace fa;
  if (S_q <= 0 || S_kv <= 0 || H < 1 || Hkv < 1 || H % Hkv) return 1;
  const int group = H / Hkv, sms = std::max(1, device_sm_count());
  const long nq = (S_q + BQ - 1) / BQ, tiles = (S_kv + BN - 1) / BN;
  long steps = 0;                                                 // query tiles of one head, over its K/V tiles
  for (long n = 0; n < tiles; ++n) steps += nq - (causal ? n * (BN / BQ) : 0);
  int best = 1;
  double best_t = 0;
  for (int parts = 1; parts <= group; ++parts) {
    if (group % parts) continue;
    const double blocks = (double)tiles * Hkv * B * parts, heavy = (double)nq * (group / parts) + 6;
    const double all = ((double)steps * H * B + 6 * blocks) / sms;
    const double waves = causal ? 0 : heavy * std::ceil(blocks / sms);            // equal blocks: whole rounds
    const double t = std::max({heavy, all + (causal ? heavy / 4 : 0), waves}) + (parts > 1 ? 0.03 * blocks : 0);
    if (parts == 1 || t < best_t * (best == 1 ? 0.95 : 1.0)) { best = parts; best_t = t; }
  }
  return best;
}

int flash_attn_bwd_query_tiles(int S_q) { return (S_q + fa::BQ - 1) / fa::BQ; }

// `turnstile`: null, or one counter per (batch, head, query tile) for dQ in a fixed order (fa_bwd_kernel<true>)
void flash_attn_bwd(const void* go, const void* q, const void* k, const void* v, const void* o, const float* lse,
                    const float* dlse, void* dq,
                    void* dk, void* dv, float* stats, float* dq_acc, float* kv_part, unsigned* turnstile, int parts, int B, int S_q, int S_kv, int H,
                    int Hkv, int S_pad, const long* gs, const long* qs, const long* ks, const long* vs, const long* os,
                    const long* dqs, const long* dks, const long* dvs, float scale, bool causal, cudaStream_t st) {
  using namespace fa;
  if (causal && S_q != S_kv) nxd_throw("attention: causal needs S_q == S_kv", __FILE__, __LINE__);
  BwdParams p;
  p.S_q = S_q; p.S_kv = S_kv; p.H = H; p.Hkv = Hkv; p.B = B; p.S_pad = S_pad;
  const CUtensorMap tq = view_tmap(View{q, B, S_q, H, qs[0], qs[1], qs[2]}, p.q, BQ);
  const CUtensorMap tg = view_tmap(View{go, B, S_q, H, gs[0], gs[1], gs[2]}, p.g, BQ);
  const CUtensorMap tk = view_tmap(View{k, B, S_kv, Hkv, ks[0], ks[1], ks[2]}, p.k);
  const CUtensorMap tv = view_tmap(View{v, B, S_kv, Hkv, vs[0], vs[1], vs[2]}, p.v);
  p.dk_sb = dks[0]; p.dk_ss = dks[1]; p.dk_sh = dks[2];
  p.dv_sb = dvs[0]; p.dv_ss = dvs[1]; p.dv_sh = dvs[2];
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.causal = causal ? 1 : 0;
  p.stats = stats; p.stats_stride = (long)B * H * S_pad + 64;
  p.dq_acc = dq_acc;
  p.parts = parts; p.kv_part = kv_part;
  const bool det = turnstile != nullptr;
  p.turnstile = turnstile;
  if (det) NXD_CUDA_CHECK(cudaMemsetAsync(turnstile, 0, (size_t)B * H * flash_attn_bwd_query_tiles(S_q) * sizeof(unsigned), st));
  {
    const long rows = (long)B * H * S_pad;
    // an ordinary launch: the main kernel loads K, V, Q and dO before it waits for this one, so they have to be there when this one starts
    fa_bwd_prep_kernel<<<(unsigned)((rows + 15) / 16), 256, 0, st>>>((const __nv_bfloat16*)o, (const __nv_bfloat16*)go, lse, dlse, stats,
                                                                     dq_acc, p.stats_stride, B, S_q, H, S_pad, os[0], os[1], os[2], gs[0],
                                                                     gs[1], gs[2], scale);
  }
  NXD_ALLOW_SMEM(fa_bwd_kernel<false>, kSmemBwd);
  NXD_ALLOW_SMEM(fa_bwd_kernel<true>, kSmemBwd);
  const long head_bytes = (long)S_q * HD * 8 * (H / Hkv / parts); // Q, dO and fp32 dQ of one block's query heads
  p.group_bh = (int)std::min<long>((long)Hkv * parts * B, std::max<long>(1, (64l << 20) / std::max<long>(1, head_bytes)));
  const unsigned grid = (unsigned)((S_kv + BN - 1) / BN * (long)Hkv * parts * B);
  NXD_CUDA_CHECK(cudaGetLastError());
  launch_dependent(det ? fa_bwd_kernel<true> : fa_bwd_kernel<false>, grid, kThreadsBwd, kSmemBwd, st, tq, tk, tv, tg, (__nv_bfloat16*)dk,
                   (__nv_bfloat16*)dv, p);
  {
    const long n = (long)B * H * S_q * 16;
    launch_dependent(fa_bwd_dq_out_kernel, (unsigned)((n + 255) / 256), 256, 0, st, (const float*)dq_acc, (__nv_bfloat16*)dq, B, S_q, H, S_pad, dqs[0],
                     dqs[1], dqs[2]);
  }
  if (parts > 1) {
    const long n = 2l * B * Hkv * S_kv * 16;
    launch_dependent(fa_bwd_kv_out_kernel, (unsigned)((n + 255) / 256), 256, 0, st, (const float*)kv_part, (__nv_bfloat16*)dk, (__nv_bfloat16*)dv, B,
                     S_kv, Hkv, parts, dks[0], dks[1], dks[2], dvs[0], dvs[1], dvs[2]);
  }
}

}  // namespace nxd

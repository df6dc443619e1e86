// bf16 GEMM, CTA-pair variant: two SMs of a cluster cooperate on one 256×256 output tile with
// tcgen05.mma.cta_group::2 (UMMA M=256, N=256, K=16).  Each CTA stages its own 128 rows of A and HALF of the B tile
// (128 of the 256 N-rows), so per-CTA shared-memory fill and L2→SMEM traffic for B halve versus the single-CTA kernel
// and the ring deepens to 6 stages × 32 KB.  The leader CTA (cluster rank 0) issues every MMA; completion is
// multicast to both CTAs' barriers with tcgen05.commit…multicast::cluster; each CTA drains its own 128 TMEM lanes.
//
//   warp 0  TMA producer (both CTAs; cta_group::2 loads signal the leader's full barrier)
//   warp 1  MMA issuer   (leader only) + TMEM allocator (both, cta_group::2)
//   warps 2-5 epilogue   (both)
#include <cuda.h>

#include <algorithm>
#include <cstdlib>
#include <string>

#include "common.cuh"
#include "kernels.h"
#include "sm100_ptx.cuh"
#include "gemm2cta.cuh"

namespace nxd {
namespace g2 {

// Grouped (routed experts) modes.  MODE 3: every `block_rows`-row block of A (a multiple of 256: a pair's tile stays inside one
// block) meets the weights of one expert, `b_rows` rows further down the stacked B per expert; `used_blocks` (device, may be
// null) bounds the blocks that hold tokens.  MODE 4 (weight gradients): one output matrix per expert, summed over that
// expert's row blocks [seg[e], seg[e + 1]); an expert without tokens gets zeros.  With `slot_token` (token of each row, -1: padding, behind all
// rows with one) the k-blocks of an expert's last row block that hold padding alone, zeros, are left out: 96 of 1150 rows an expert on average
// with 1024 tokens each.
constexpr int kExpertRows = 4;       // row tiles that go through the columns together: about one expert's (with 16, two per cent slower)
struct Group {
  const int* block_expert;
  const int* seg;
  const int* used_blocks;
  int block_rows, b_rows, groups;
  const int* slot_token;
};

// The tiles of the last, partial round of pairs (`tiles` of them) are split along K over `splits`
// pairs each, `kb_per` k-blocks apiece; their fp32 partials go to a workspace [tiles * splits][256][columns of a tile] that gemm_tail_kernel
// sums.  80 tiles on 74 pairs took two tiles' time for 1.08 of work.
struct Tail { int tiles, splits, kb_per; };

// MODE 0: one product.  MODE 5: SwiGLU of the product with [gate; up] weights; a tile's 256 columns are 128 gates (the first CTA's half of B) and the
// 128 ups that belong to them (the second's), its outputs 128 columns; N counts outputs.  MODE 6: the products are kept too (a backward
// pass needs them).  MODE 7: routed experts with [gate up] weights, the products kept if `accumulate`.
__host__ __device__ constexpr bool gated(int mode) { return mode >= 5 && mode <= 7; }
__host__ __device__ constexpr bool experts(int mode) { return mode == 3 || mode == 7; }
__host__ __device__ constexpr bool whole(int mode) { return mode == 0 || mode == 5 || mode == 6; }

// one unit of work of a pair: an output tile and its range of k-blocks; `part`: a split of a tail tile, number `mat`
struct Unit { int m_blk, n_blk, mat, kb0, kb1; bool part; };

template <int MODE>
NXD_DEVICE Unit unit_of(int unit, int num_tiles, int tiles_m, int tiles_n, int num_kb, int kb_per, const Group& g, const Tail& tail) {
  Unit u;
  u.mat = 0;
  u.part = false;
  if constexpr (whole(MODE)) {
    const int x = unit - (num_tiles - tail.tiles);
    if (tail.tiles > 0 && x >= 0) {                        // never together with split_k
      u.part = true;
      u.mat = x;
      tile_coords(num_tiles - tail.tiles + x / tail.splits, tiles_m, tiles_n, raster_rows(tiles_m), u.m_blk, u.n_blk);
      u.kb0 = x % tail.splits * tail.kb_per;
      u.kb1 = min(num_kb, u.kb0 + tail.kb_per);
      return u;
    }
  }
  if constexpr (MODE == 4) {
    const int per = tiles_m * tiles_n;
    u.mat = unit / per;
    tile_coords(unit - u.mat * per, tiles_m, tiles_n, kExpertRows, u.m_blk, u.n_blk);
    u.kb0 = g.seg[u.mat] * (g.block_rows / BK);
    u.kb1 = g.seg[u.mat + 1] * (g.block_rows / BK);
    if (g.slot_token) {                                    // the first row of a k-block tells whether it has any (the first k-block of a row block has)
      const int per_block = g.block_rows / BK;
      int kept = u.kb0 == u.kb1 ? 0 : 1;
      for (int i = 1; i < per_block; ++i) kept += u.kb0 < u.kb1 && g.slot_token[(u.kb1 - per_block + i) * BK] >= 0;
      u.kb1 += kept - (u.kb0 == u.kb1 ? 0 : per_block);
    }
  } else {
    const int ks = unit / num_tiles;
    tile_coords(unit - ks * num_tiles, tiles_m, tiles_n, whole(MODE) ? raster_rows(tiles_m) : kExpertRows, u.m_blk, u.n_blk);
    u.kb0 = ks * kb_per;
    u.kb1 = min(num_kb, (ks + 1) * kb_per);
  }
  return u;
}

// Stages, shared memory and accumulators for tiles of TN columns: 256, or 128 where an output has too few of those to fill the chip.
template <int TN>
struct Shape {
  static constexpr int kHalfN = TN / 2, kBytesB = kHalfN * BK * 2, kBytes = kABytes + kBytesB, kRing = TN == 256 ? kStages : 8;
  static constexpr int kEpi = kRing * kBytes, kBars = kEpi + kEpiBufs * kEpiSlabBytes, kShared = kBars + 1024 + 256;
  static_assert(kShared <= 232448, "exceeds the 227 KB of dynamic shared memory per CTA");
};

template <bool A_KMAJOR, bool B_KMAJOR, typename OutT, int MODE, int TN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_bf16_2cta_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                      const __grid_constant__ CUtensorMap tma_out, const __grid_constant__ CUtensorMap tma_part,
                      const __grid_constant__ CUtensorMap tma_keep, OutT* out, int M, int N, int K, int accumulate, int split_k, const Group grp, const Tail tail) {
  // accumulate: 0 store, 1 add to what is there.  split_k > 1 (fp32 outputs): that many pairs share one output tile, each sums
  // a K range and adds its partial — for weight gradients whose output has too few tiles to fill the 74 pairs while
  // K = tokens is long.  fp32 outputs always leave through TMA (stored or added in memory), bf16 ones unless they accumulate.
  using S = Shape<TN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + S::kBars);
  uint32_t* tmem_slot = (uint32_t*)(bars + 2 * S::kRing + 2 * kAcc);
  const uint32_t bar_full = smem_u32(bars), bar_empty = smem_u32(bars + S::kRing);
  const uint32_t bar_tfull = smem_u32(bars + 2 * S::kRing), bar_tempty = smem_u32(bars + 2 * S::kRing + kAcc);
  const uint32_t smem_base = smem_u32(smem);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();
  const bool leader = cta == 0;
  int tiles_m = (M + TILE_M - 1) / TILE_M;
  constexpr int kCols = gated(MODE) ? TN / 2 : TN;             // outputs of a tile
  const int tiles_n = (N + kCols - 1) / kCols;
  if constexpr (experts(MODE)) { if (grp.used_blocks) tiles_m = min(tiles_m, *grp.used_blocks * (grp.block_rows / TILE_M)); }
  const int num_tiles = (MODE == 4 ? grp.groups : 1) * tiles_m * tiles_n;
  const int num_kb = (K + BK - 1) / BK;
  const int kb_per = (num_kb + split_k - 1) / split_k;       // k-blocks per split (host guarantees no empty split)
  const int num_units = num_tiles * split_k + tail.tiles * (tail.splits - 1);
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;

  if (warp == 0 && lane == 0) {
    prefetch_tmap(&tma_a);
    prefetch_tmap(&tma_b);
    for (int i = 0; i < S::kRing; ++i) {
      mbar_init(bar_full + 8 * i, 2);     // leader: own arrive.expect_tx + peer's remote arrive
      mbar_init(bar_empty + 8 * i, 1);    // one multicast tcgen05.commit
    }
    for (int i = 0; i < kAcc; ++i) {
      mbar_init(bar_tfull + 8 * i, 1);
      mbar_init(bar_tempty + 8 * i, 2 * 128);   // epilogue threads of both CTAs (used on the leader)
    }
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 1) { tcgen05_alloc_2cta(smem_u32(tmem_slot), kAcc * TN); tcgen05_relinquish_2cta(); }
  tcgen05_fence_before();
  cluster_sync_all();               // barriers of both CTAs are initialised before any remote arrive
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if constexpr (whole(MODE)) {
    pdl_trigger();                                           // behind the allocation (launch_dependent)
    pdl_wait();                                              // all before this has run beside the end of the kernel before
  }

  if (warp == 0) {
    // ===== TMA producer (both CTAs) =====
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      for (int unit = pair; unit < num_units; unit += num_pairs) {
        const Unit u = unit_of<MODE>(unit, num_tiles, tiles_m, tiles_n, num_kb, kb_per, grp, tail);
        const int m0 = u.m_blk * TILE_M + (int)cta * CTA_M;
        const int n0 = gated(MODE) ? u.n_blk * kCols + (int)cta * N : u.n_blk * TN + (int)cta * S::kHalfN;
        int b_off = 0;
        if constexpr (experts(MODE)) b_off = grp.block_expert[u.m_blk * TILE_M / grp.block_rows] * grp.b_rows;
        for (int kb = u.kb0; kb < u.kb1; ++kb) {
          mbar_wait(bar_empty + 8 * stage, phase ^ 1);
          const uint32_t full = bar_full + 8 * stage;          // same offset in the leader's smem
          if (leader) mbar_expect_tx(full, 2 * S::kBytes);
          else mbar_arrive_cluster(mapa_shared(full, 0));
          const uint32_t sa = smem_base + stage * S::kBytes, sb = sa + kABytes;
          const int k0 = kb * BK;
          if constexpr (A_KMAJOR) {
            tma_load_2d_2cta(sa, &tma_a, full, k0, m0);                          // box {64 k, 128 m}
          } else {
#pragma unroll
            for (int j = 0; j < CTA_M / 64; ++j) tma_load_2d_2cta(sa + j * 8192, &tma_a, full, m0 + j * 64, k0);
          }
          if constexpr (B_KMAJOR) {
            tma_load_2d_2cta(sb, &tma_b, full, k0, b_off + n0);                  // box {64 k, 128 n}
          } else {
#pragma unroll
            for (int j = 0; j < S::kHalfN / 64; ++j) tma_load_2d_2cta(sb + j * 8192, &tma_b, full, n0 + j * 64, b_off + k0);
          }
          if (++stage == S::kRing) { stage = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ===== MMA issuer (leader CTA only) =====
    if (leader) {                                          // all lanes; the helpers elect one
      constexpr uint32_t idesc = make_idesc(!A_KMAJOR, !B_KMAJOR, TILE_M, TN);
      int stage = 0; uint32_t phase = 0; int as = 0; uint32_t aphase = 0;
      for (int unit = pair; unit < num_units; unit += num_pairs) {
        const Unit u = unit_of<MODE>(unit, num_tiles, tiles_m, tiles_n, num_kb, kb_per, grp, tail);
        mbar_wait(bar_tempty + 8 * as, aphase ^ 1);
        tcgen05_fence_after();
        const uint32_t tmem_d = tmem_base + as * TN;
        for (int kb = u.kb0; kb < u.kb1; ++kb) {
          mbar_wait(bar_full + 8 * stage, phase);
          tcgen05_fence_after();
          const uint32_t sa = smem_base + stage * S::kBytes, sb = sa + kABytes;
          mma4_commit_2cta<A_KMAJOR ? 2 : 128, B_KMAJOR ? 2 : 128>(tmem_d, A_KMAJOR ? make_smem_desc(sa, 16, 1024) : make_smem_desc(sa, 8192, 1024),
                                                                   B_KMAJOR ? make_smem_desc(sb, 16, 1024) : make_smem_desc(sb, 8192, 1024), idesc,
                                                                   kb != u.kb0 ? 1u : 0u, bar_empty + 8 * stage);
          if (++stage == S::kRing) { stage = 0; phase ^= 1; }
        }
        tcgen05_commit_2cta_e(bar_tfull + 8 * as, 0b11);       // accumulators ready in both CTAs
        if (++as == kAcc) { as = 0; aphase ^= 1; }
      }
    }
    __syncwarp();
  } else {
    // ===== epilogue (both CTAs; own 128 TMEM lanes) =====
    const int q = warp & 3;
    const uint32_t tempty_leader = mapa_shared(bar_tempty, 0);
    const bool issuer = threadIdx.x == 64;
    uint32_t slab_ctr = 0;
    int as = 0; uint32_t aphase = 0;
    for (int unit = pair; unit < num_units; unit += num_pairs) {
      const Unit u = unit_of<MODE>(unit, num_tiles, tiles_m, tiles_n, num_kb, kb_per, grp, tail);
      mbar_wait(bar_tfull + 8 * as, aphase);
      tcgen05_fence_after();
      const int n0 = u.n_blk * kCols, row0 = u.m_blk * TILE_M + (int)cta * CTA_M;
      const uint32_t acc = tmem_base + ((uint32_t)(q * 32) << 16) + as * TN;
      const bool empty = MODE == 4 && u.kb0 == u.kb1;
      if (whole(MODE) && u.part) {
        epilogue_tile_tma_f32<TN>(acc, smem_base + S::kEpi, &tma_part, (int)cta * CTA_M, u.mat, 0, TN, q, lane, issuer, slab_ctr,
                              false, false);
      } else if constexpr (gated(MODE)) {
        if (MODE == 6 || (MODE == 7 && accumulate)) {
          epilogue_tile_tma<false, TN / 2>(acc, smem_base + S::kEpi, &tma_keep, row0, n0, 2 * N, q, lane, issuer, slab_ctr);
          epilogue_tile_tma<false, TN / 2>(acc + TN / 2, smem_base + S::kEpi, &tma_keep, row0, N + n0, 2 * N, q, lane, issuer, slab_ctr);
        }
        epilogue_tile_swiglu(acc, smem_base + S::kEpi, &tma_out, row0, n0, q, lane, issuer, slab_ctr);
      } else if constexpr (sizeof(OutT) == 4) {
        epilogue_tile_tma_f32<TN>(acc, smem_base + S::kEpi, &tma_out, row0, u.mat, n0, N, q, lane, issuer, slab_ctr,
                              accumulate || split_k > 1, empty);
      } else if (!accumulate) {
        epilogue_tile_tma<MODE == 4, TN>(acc, smem_base + S::kEpi, &tma_out, row0, n0, N, q, lane, issuer, slab_ctr, u.mat, empty);
      } else {
        const int row = row0 + q * 32 + lane;
        OutT* orow = out + ((size_t)u.mat * M + row) * N;
        const bool row_ok = row < M;
#pragma unroll 1
        for (int c = 0; c < TN / 32; ++c) {
          uint32_t r[32];
          tcgen05_ld_32x32(acc + c * 32, r);
          tcgen05_wait_ld();
          const int col0 = n0 + c * 32;
          if (row_ok && col0 < N && !empty) store_chunk<OutT>(orow, col0, N, r, accumulate);
        }
      }
      tcgen05_fence_before();
      mbar_arrive_cluster(tempty_leader + 8 * as);   // leader's barrier collects both CTAs' epilogues
      if (++as == kAcc) { as = 0; aphase ^= 1; }
    }
    if (issuer) bulk_wait<0>();      // staging smem must outlive the last stores' reads; output complete at kernel end
  }

  tcgen05_fence_before();
  cluster_sync_all();               // peer must be done with our smem/TMEM before teardown
  if (warp == 1) { __syncwarp(); tcgen05_dealloc_2cta(tmem_base, kAcc * TN); }
}

// out tile (+)= sum of its splits' partials, in order: one thread per 8 columns of a row
// GATE: tiles of 128 gates and their 128 ups; SwiGLU of the two sums, 8 of 128 columns a thread; `keep`, if any: the sums, [M, 2 N]
template <typename OutT, int TN, bool GATE = false>
__global__ void __launch_bounds__(256) gemm_tail_kernel(const float* part, OutT* out, int M, int N, int first,
                                                        int tiles_m, int tiles_n, int splits, int accumulate, OutT* keep) {
  pdl_trigger();
  pdl_wait();
  constexpr int kCols = GATE ? TN / 2 : TN, kPer = kCols / 8;      // outputs of a tile, threads of a row
  const int t = blockIdx.y, row = blockIdx.x * (256 / kPer) + threadIdx.x / kPer, col = threadIdx.x % kPer * 8;
  int m_blk, n_blk;
  tile_coords(first + t, tiles_m, tiles_n, raster_rows(tiles_m), m_blk, n_blk);
  const int gr = m_blk * TILE_M + row, gc = n_blk * kCols + col;
  if (gr >= M || gc >= N) return;                          // N is a multiple of 8
  float a[8] = {}, b[GATE ? 8 : 1] = {};
  auto sum = [&](float* v, int c) {
    const float* src = part + ((size_t)t * splits * TILE_M + row) * TN + c;
#pragma unroll 4
    for (int s = 0; s < splits; ++s) {
      const float4 x = *reinterpret_cast<const float4*>(src + (size_t)s * TILE_M * TN);
      const float4 y = *reinterpret_cast<const float4*>(src + (size_t)s * TILE_M * TN + 4);
      v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w; v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
    }
  };
  sum(a, col);
  if constexpr (GATE) {
    static_assert(sizeof(OutT) == 2);
    sum(b, kCols + col);
    if (keep) {
      Pack16<OutT> gate, up;
#pragma unroll
      for (int j = 0; j < 8; ++j) { gate.set(j, a[j]); up.set(j, b[j]); }
      OutT* row_of = keep + (size_t)gr * 2 * N + gc;
      gate.store(row_of);
      up.store(row_of + N);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = silu_mul_bf16(a[j], b[j]);
  }
  OutT* dst = out + (size_t)gr * N + gc;
#pragma unroll
  for (int v = 0; v < 8; v += Pack16<OutT>::N) {
    Pack16<OutT> o;
    if (accumulate) o.load(dst + v);
#pragma unroll
    for (int j = 0; j < Pack16<OutT>::N; ++j) o.set(j, accumulate ? a[v + j] + o.f(j) : a[v + j]);
    o.store(dst + v);
  }
}


// =====================================================================================================
// Tensor-parallel fused variants on the CTA-pair kernel (no NCCL call on these paths).
//   MODE 1  all-gather → GEMM   : the first `comm_ctas` CTAs push this rank's A shard to every peer's symmetric buffer
//                                 (coalesced 16 B × 192-thread stores over NVLink) and publish per-(source,128-row block)
//                                 flags (st.release.sys = epoch); GEMM pairs walk the row chunks in arrival order, each
//                                 CTA's TMA producer acquiring the flag of its own 128 rows first.
//   MODE 2  GEMM → reduce-scatter: GEMM pairs write bf16 partial tiles to a LOCAL buffer (L2-merged stores) and bump a
//                                 local per-row-block counter; comm CTAs wait for a row block to be complete and push it to
//                                 the owner's staging slot as full 512 B rows (NVLink-friendly bursts, decoupled from the
//                                 MMA epilogue), then publish the owner's flag; finally every CTA becomes a reducer that
//                                 sums the world partials of its rank's rows in fp32.
// =====================================================================================================
struct TpComm {
  int mode, rank, world;
  const int64_t* peer_bufs;
  const int64_t* peer_flags;
  long buf_offset;
  int flag_offset;
  uint32_t epoch;
  int comm_ctas;
  int rows_per_rank;
  const void* a_local;
  void* rs_out;
  uint32_t* tile_done;
  uint32_t* gemm_done;
  uint32_t gemm_done_target;
  int push_tma;            // 0: register-staged 16-byte copies; 1: TMA bulk copies through smem, per item; 2: streaming across items
};
constexpr int kMaxRowBlocks = 64;


template <int MODE>
NXD_DEVICE void tp_tile_coords(int tile, int tiles_n, const TpComm& c, int& m_blk, int& n_blk) {
  const int mb_per_rank = c.rows_per_rank / TILE_M;           // 256-row blocks per rank
  const int per_chunk = mb_per_rank * tiles_n;
  const int step = tile / per_chunk;
  const int in = tile - step * per_chunk;
  const int chunk = MODE == 1 ? (c.rank - step + c.world) % c.world : (c.rank + 1 + step) % c.world;
  m_blk = chunk * mb_per_rank + in % mb_per_rank;
  n_blk = in / mb_per_rank;
}

// copy `bytes` (multiple of 16) with all threads of the CTA.  16 independent 16-byte loads are in flight per thread
// (48 KB per CTA) before the first store issues: NVLink/L2 latency is ~1-2 us, so bytes-in-flight is what sets the
// per-CTA copy bandwidth.
NXD_DEVICE void cta_copy16(uint8_t* dst, const uint8_t* src, size_t bytes) {
  constexpr int U = 16;
  const size_t nvec = bytes / 16;
  const uint4* s4 = (const uint4*)src;
  uint4* d4 = (uint4*)dst;
  size_t i = threadIdx.x;
  for (; i + (U - 1) * kThreads < nvec; i += U * kThreads) {
    uint4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = s4[i + u * kThreads];
#pragma unroll
    for (int u = 0; u < U; ++u) d4[i + u * kThreads] = v[u];
  }
  for (; i < nvec; i += kThreads) d4[i] = s4[i];
}

// TMA push: one thread streams `bytes` (multiple of 16) from local global memory to a peer address through this CTA's
// (otherwise idle) GEMM smem ring: cp.async.bulk global→smem (mbarrier completion) then smem→peer-global (bulk group).
// Five 32 KB loads and one or two stores are in flight per CTA without using a single data register, which is what the
// register-staged copy (48 KB in flight, one fence per block) could not do.  `phases` carries the ring's barrier parities
// across calls.  Barriers: the comm CTA borrows bar_empty[] (count 1) of the GEMM pipeline it never runs.
NXD_DEVICE void tma_push(uint8_t* dst, const uint8_t* src, size_t bytes, uint32_t smem_base, uint32_t bar0, uint32_t& phases) {
  constexpr uint32_t CH = (uint32_t)kStageBytes;
  constexpr int NST = kStages;
  const int n = (int)((bytes + CH - 1) / CH);
  auto chunk_bytes = [&](int c) { return (uint32_t)min((size_t)CH, bytes - (size_t)c * CH); };
  auto load = [&](int c) {
    const int st = c % NST;
    const uint32_t b = bar0 + 8 * st, nb = chunk_bytes(c);
    mbar_expect_tx(b, nb);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_base + st * CH), "l"(src + (size_t)c * CH), "r"(nb), "r"(b) : "memory");
  };
  for (int c = 0; c < n && c < NST; ++c) load(c);
  for (int c = 0; c < n; ++c) {
    const int st = c % NST;
    mbar_wait(bar0 + 8 * st, (phases >> st) & 1u);
    phases ^= 1u << st;
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                 ::"l"(dst + (size_t)c * CH), "r"(smem_base + st * CH), "r"(chunk_bytes(c)) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    if (c >= 1 && c - 1 + NST < n) {
      asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");     // store c-1 has drained its stage
      load(c - 1 + NST);
    }
  }
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  asm volatile("fence.proxy.async.global;" ::: "memory");
}

// Streaming variant of tma_push (push_tma == 2, opt-in until measured): the smem ring is kept full ACROSS the CTA's items — no
// drain between 1 MB blocks.  Item k's flag is published as soon as all of its store groups have COMPLETED, which
// `cp.async.bulk.wait_group NST` guarantees for every group older than the newest NST ones; only when the next item is not
// ready yet (GEMM→RS) or at the very end is the pipeline drained.  `item(k, src, dst, flag)` yields the k-th item of this CTA,
// `ready(k)` blocks until its source is complete (no-op for the all-gather).
template <typename ItemFn, typename ReadyFn, typename PendingFn>
NXD_DEVICE void tma_push_stream(int n_items, size_t item_bytes, uint32_t epoch, uint32_t smem_base, uint32_t bar0,
                                uint32_t& phases, ItemFn item, ReadyFn ready, PendingFn is_ready) {
  constexpr uint32_t CH = (uint32_t)kStageBytes;
  constexpr int NST = kStages;
  const int cpi = (int)((item_bytes + CH - 1) / CH);          // chunks per item
  const long total = (long)n_items * cpi;
  int next_flag = 0;                                          // items [0, next_flag) have been published
  auto publish_upto = [&](int k_end) {                        // caller guarantees completion of those items' stores
    if (next_flag >= k_end) return;
    asm volatile("fence.proxy.async.global;" ::: "memory");
    __threadfence_system();
    for (; next_flag < k_end; ++next_flag) {
      const uint8_t* s_; uint8_t* d_; uint32_t* f_;
      item(next_flag, s_, d_, f_);
      st_release_sys(f_, epoch);
    }
  };
  auto chunk_bytes = [&](int c) { return (uint32_t)min((size_t)CH, item_bytes - (size_t)c * CH); };
  long issued = 0;                                            // loads issued so far (global chunk index)
  int ready_upto = 0;                                         // items [0, ready_upto) are known to be loadable
  auto load = [&](long g) {
    const int k = (int)(g / cpi), c = (int)(g % cpi);
    const uint8_t* s_; uint8_t* d_; uint32_t* f_;
    item(k, s_, d_, f_);
    const int st = (int)(g % NST);
    const uint32_t b = bar0 + 8 * st, nb = chunk_bytes(c);
    mbar_expect_tx(b, nb);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_base + st * CH), "l"(s_ + (size_t)c * CH), "r"(nb), "r"(b) : "memory");
  };
  for (long g = 0; g < total; ++g) {
    // keep up to NST-1 loads ahead of the store cursor; never load from an item that is not ready
    while (issued < total && issued < g + NST - 1 + (g == 0 ? 1 : 0)) {
      const int k = (int)(issued / cpi);
      if (k >= ready_upto) {
        if (!is_ready(k)) {
          if (issued > g) break;                              // there is still loaded work to store: come back later
          asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // nothing in flight to overlap with: drain, publish, block
          publish_upto((int)(g / cpi));
          ready(k);
        }
        asm volatile("fence.proxy.async.global;" ::: "memory");       // generic-proxy producer writes → async-proxy reads
        ready_upto = k + 1;
      }
      if (issued >= NST) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(1) : "memory");   // stage reuse: its old store has drained
      load(issued++);
    }
    const int k = (int)(g / cpi), c = (int)(g % cpi), st = (int)(g % NST);
    const uint8_t* s_; uint8_t* d_; uint32_t* f_;
    item(k, s_, d_, f_);
    mbar_wait(bar0 + 8 * st, (phases >> st) & 1u);
    phases ^= 1u << st;
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                 ::"l"(d_ + (size_t)c * CH), "r"(smem_base + st * CH), "r"(chunk_bytes(c)) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    // every group older than the newest NST has fully completed after this wait → items that ended there can be flagged
    asm volatile("cp.async.bulk.wait_group %0;" ::"n"(NST) : "memory");
    const long done_upto = g - NST;                           // global chunk index whose store is certainly complete
    if (done_upto >= 0) publish_upto((int)((done_upto + 1) / cpi));
  }
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  publish_upto(n_items);
}

template <bool A_KMAJOR, bool B_KMAJOR, int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_bf16_2cta_tp_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                         const __grid_constant__ CUtensorMap tma_a_local, __nv_bfloat16* __restrict__ out, int M, int N,
                         int K, TpComm comm) {
  using OutT = __nv_bfloat16;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + kBarOffset);
  uint32_t* tmem_slot = (uint32_t*)(bars + 2 * kStages + 2 * kAcc);
  const uint32_t bar_full = smem_u32(bars), bar_empty = smem_u32(bars + kStages);
  const uint32_t bar_tfull = smem_u32(bars + 2 * kStages), bar_tempty = smem_u32(bars + 2 * kStages + kAcc);
  const uint32_t smem_base = smem_u32(smem);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();
  const bool leader = cta == 0;
  const int tiles_m = (M + TILE_M - 1) / TILE_M, tiles_n = (N + TILE_N - 1) / TILE_N;
  const int num_tiles = tiles_m * tiles_n;
  const int num_kb = (K + BK - 1) / BK;
  const bool is_comm = (int)blockIdx.x < comm.comm_ctas;
  const int pair = ((int)blockIdx.x - comm.comm_ctas) >> 1, num_pairs = ((int)gridDim.x - comm.comm_ctas) >> 1;
  const int blk128_per_rank = comm.rows_per_rank / CTA_M;

  if (warp == 0 && lane == 0) {
    prefetch_tmap(&tma_a);
    prefetch_tmap(&tma_b);
    prefetch_tmap(&tma_a_local);
    for (int i = 0; i < kStages; ++i) { mbar_init(bar_full + 8 * i, 2); mbar_init(bar_empty + 8 * i, 1); }
    for (int i = 0; i < kAcc; ++i) { mbar_init(bar_tfull + 8 * i, 1); mbar_init(bar_tempty + 8 * i, 2 * 128); }
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 1) { tcgen05_alloc_2cta(smem_u32(tmem_slot), kTmemCols); tcgen05_relinquish_2cta(); }
  tcgen05_fence_before();
  cluster_sync_all();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (is_comm) {
    uint32_t push_phases = 0;
    if constexpr (MODE == 1) {
      // ---- all-gather pusher: (destination step, 128-row block) items.  The local chunk is NOT copied: GEMM tiles of
      //      the own chunk read the shard in place through `tma_a_local` and start immediately. -------------------
      const int items = (comm.world - 1) * blk128_per_rank;
      const size_t blk_bytes = (size_t)CTA_M * K * 2;
      if (comm.push_tma == 2) {
        if (threadIdx.x == 0) {
          const int mine = ((int)blockIdx.x < items) ? (items - 1 - (int)blockIdx.x) / comm.comm_ctas + 1 : 0;
          auto item = [&](int k, const uint8_t*& src, uint8_t*& d, uint32_t*& f) {
            const int it = (int)blockIdx.x + k * comm.comm_ctas;
            const int step = it / blk128_per_rank + 1, mb = it % blk128_per_rank;
            const int dst = (comm.rank + step) % comm.world;
            src = (const uint8_t*)comm.a_local + (size_t)mb * blk_bytes;
            d = (uint8_t*)comm.peer_bufs[dst] + comm.buf_offset + ((size_t)comm.rank * blk128_per_rank + mb) * blk_bytes;
            f = (uint32_t*)comm.peer_flags[dst] + comm.flag_offset + comm.rank * kMaxRowBlocks + mb;
          };
          tma_push_stream(mine, blk_bytes, comm.epoch, smem_base, bar_empty, push_phases, item, [](int) {}, [](int) { return true; });
        }
      } else
      for (int it = blockIdx.x; it < items; it += comm.comm_ctas) {
        const int step = it / blk128_per_rank + 1, mb = it % blk128_per_rank;
        const int dst = (comm.rank + step) % comm.world;
        const uint8_t* src = (const uint8_t*)comm.a_local + (size_t)mb * blk_bytes;
        uint8_t* d = (uint8_t*)comm.peer_bufs[dst] + comm.buf_offset +
                     ((size_t)comm.rank * blk128_per_rank + mb) * blk_bytes;
        if (comm.push_tma) {
          if (threadIdx.x == 0) {
            tma_push(d, src, blk_bytes, smem_base, bar_empty, push_phases);
            __threadfence_system();
            st_release_sys((uint32_t*)comm.peer_flags[dst] + comm.flag_offset + comm.rank * kMaxRowBlocks + mb, comm.epoch);
          }
        } else {
          cta_copy16(d, src, blk_bytes);
          __threadfence_system();
          __syncthreads();
          if (threadIdx.x == 0)
            st_release_sys((uint32_t*)comm.peer_flags[dst] + comm.flag_offset + comm.rank * kMaxRowBlocks + mb, comm.epoch);
        }
      }
    } else {
      // ---- reduce-scatter pusher: ship finished row blocks of remote chunks to their owners -------------------
      const int items = (comm.world - 1) * blk128_per_rank;
      const size_t blk_bytes = (size_t)CTA_M * N * 2;
      if (comm.push_tma == 2) {
        if (threadIdx.x == 0) {
          const int mine = ((int)blockIdx.x < items) ? (items - 1 - (int)blockIdx.x) / comm.comm_ctas + 1 : 0;
          auto gblk_of = [&](int k, int& owner, int& mb) {
            const int it = (int)blockIdx.x + k * comm.comm_ctas;
            const int step = it / blk128_per_rank;
            mb = it % blk128_per_rank;
            owner = (comm.rank + 1 + step) % comm.world;
            return owner * blk128_per_rank + mb;
          };
          auto item = [&](int k, const uint8_t*& src, uint8_t*& d, uint32_t*& f) {
            int owner, mb;
            const int gblk = gblk_of(k, owner, mb);
            src = (const uint8_t*)out + (size_t)gblk * blk_bytes;
            d = (uint8_t*)comm.peer_bufs[owner] + comm.buf_offset + ((size_t)comm.rank * blk128_per_rank + mb) * blk_bytes;
            f = (uint32_t*)comm.peer_flags[owner] + comm.flag_offset + comm.rank * kMaxRowBlocks + mb;
          };
          auto is_ready = [&](int k) {
            int owner, mb;
            const int gblk = gblk_of(k, owner, mb);
            if (ld_acquire_gpu(comm.tile_done + gblk) < (uint32_t)tiles_n) return false;
            comm.tile_done[gblk] = 0;                                  // single consumer: re-arm for the next call
            return true;
          };
          auto ready = [&](int k) { while (!is_ready(k)) __nanosleep(128); };
          tma_push_stream(mine, blk_bytes, comm.epoch, smem_base, bar_empty, push_phases, item, ready, is_ready);
        }
      } else
      for (int it = blockIdx.x; it < items; it += comm.comm_ctas) {
        const int step = it / blk128_per_rank, mb = it % blk128_per_rank;
        const int owner = (comm.rank + 1 + step) % comm.world;
        const int gblk = owner * blk128_per_rank + mb;                 // global 128-row block of the partial
        if (threadIdx.x == 0) {
          while (ld_acquire_gpu(comm.tile_done + gblk) < (uint32_t)tiles_n) __nanosleep(128);
          comm.tile_done[gblk] = 0;                                    // single consumer: re-arm for the next call
        }
        const uint8_t* src = (const uint8_t*)out + (size_t)gblk * blk_bytes;
        uint8_t* d = (uint8_t*)comm.peer_bufs[owner] + comm.buf_offset +
                     ((size_t)comm.rank * blk128_per_rank + mb) * blk_bytes;
        if (comm.push_tma) {
          if (threadIdx.x == 0) {
            asm volatile("fence.proxy.async.global;" ::: "memory");    // epilogue (generic) writes → TMA (async proxy) reads
            tma_push(d, src, blk_bytes, smem_base, bar_empty, push_phases);
            __threadfence_system();
            st_release_sys((uint32_t*)comm.peer_flags[owner] + comm.flag_offset + comm.rank * kMaxRowBlocks + mb, comm.epoch);
          }
        } else {
          __syncthreads();
          cta_copy16(d, src, blk_bytes);
          __threadfence_system();
          __syncthreads();
          if (threadIdx.x == 0)
            st_release_sys((uint32_t*)comm.peer_flags[owner] + comm.flag_offset + comm.rank * kMaxRowBlocks + mb, comm.epoch);
        }
      }
    }
  } else if (warp == 0) {
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      for (int tile = pair; tile < num_tiles; tile += num_pairs) {
        int m_blk, n_blk;
        tp_tile_coords<MODE>(tile, tiles_n, comm, m_blk, n_blk);
        const int m0 = m_blk * TILE_M + (int)cta * CTA_M;
        const int n0 = n_blk * TILE_N + (int)cta * HALF_N;
        const CUtensorMap* amap = &tma_a;
        int a_row = m0;
        if constexpr (MODE == 1) {
          const int gblk = m0 / CTA_M;
          const int src_rank = gblk / blk128_per_rank;
          if (src_rank == comm.rank) {
            amap = &tma_a_local;                       // own shard, in place
            a_row = m0 - src_rank * comm.rows_per_rank;
          } else {
            const uint32_t* f = (const uint32_t*)comm.peer_flags[comm.rank] + comm.flag_offset +
                                src_rank * kMaxRowBlocks + (gblk % blk128_per_rank);
            wait_flag_ge(f, comm.epoch);
            fence_proxy_async_global();
          }
        }
        for (int kb = 0; kb < num_kb; ++kb) {
          mbar_wait(bar_empty + 8 * stage, phase ^ 1);
          const uint32_t full = bar_full + 8 * stage;
          if (leader) mbar_expect_tx(full, 2 * kStageBytes);
          else mbar_arrive_cluster(mapa_shared(full, 0));
          const uint32_t sa = smem_base + stage * kStageBytes, sb = sa + kABytes;
          const int k0 = kb * BK;
          if constexpr (A_KMAJOR) {
            tma_load_2d_2cta(sa, amap, full, k0, a_row);
          } else {
#pragma unroll
            for (int j = 0; j < CTA_M / 64; ++j) tma_load_2d_2cta(sa + j * 8192, amap, full, a_row + j * 64, k0);
          }
          if constexpr (B_KMAJOR) {
            tma_load_2d_2cta(sb, &tma_b, full, k0, n0);
          } else {
#pragma unroll
            for (int j = 0; j < HALF_N / 64; ++j) tma_load_2d_2cta(sb + j * 8192, &tma_b, full, n0 + j * 64, k0);
          }
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (leader && lane == 0) {
      constexpr uint32_t idesc = make_idesc(!A_KMAJOR, !B_KMAJOR, TILE_M, TILE_N);
      int stage = 0; uint32_t phase = 0; int as = 0; uint32_t aphase = 0;
      for (int tile = pair; tile < num_tiles; tile += num_pairs) {
        mbar_wait(bar_tempty + 8 * as, aphase ^ 1);
        tcgen05_fence_after();
        const uint32_t tmem_d = tmem_base + as * TILE_N;
        for (int kb = 0; kb < num_kb; ++kb) {
          mbar_wait(bar_full + 8 * stage, phase);
          tcgen05_fence_after();
          const uint32_t sa = smem_base + stage * kStageBytes, sb = sa + kABytes;
#pragma unroll
          for (int k = 0; k < BK / UK; ++k) {
            const uint64_t da = A_KMAJOR ? make_smem_desc(sa + k * 32, 16, 1024) : make_smem_desc(sa + k * 2048, 8192, 1024);
            const uint64_t db = B_KMAJOR ? make_smem_desc(sb + k * 32, 16, 1024) : make_smem_desc(sb + k * 2048, 8192, 1024);
            tcgen05_mma_f16_2cta(tmem_d, da, db, idesc, (kb | k) != 0 ? 1u : 0u);
          }
          tcgen05_commit_2cta(bar_empty + 8 * stage, 0b11);
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
        tcgen05_commit_2cta(bar_tfull + 8 * as, 0b11);
        if (++as == kAcc) { as = 0; aphase ^= 1; }
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3;
    const uint32_t tempty_leader = mapa_shared(bar_tempty, 0);
    int as = 0; uint32_t aphase = 0;
    for (int tile = pair; tile < num_tiles; tile += num_pairs) {
      int m_blk, n_blk;
      tp_tile_coords<MODE>(tile, tiles_n, comm, m_blk, n_blk);
      mbar_wait(bar_tfull + 8 * as, aphase);
      tcgen05_fence_after();
      const int row = m_blk * TILE_M + (int)cta * CTA_M + q * 32 + lane;
      const int n0 = n_blk * TILE_N;
      OutT* orow = out + (size_t)row * N;
      const bool row_ok = row < M;
#pragma unroll 1
      for (int c = 0; c < TILE_N / 32; ++c) {
        uint32_t r[32];
        tcgen05_ld_32x32(tmem_base + ((uint32_t)(q * 32) << 16) + as * TILE_N + c * 32, r);
        tcgen05_wait_ld();
        const int col0 = n0 + c * 32;
        if (row_ok && col0 < N) store_chunk<OutT>(orow, col0, N, r, 0);
      }
      tcgen05_fence_before();
      mbar_arrive_cluster(tempty_leader + 8 * as);
      if constexpr (MODE == 2) {
        __threadfence();
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (threadIdx.x == 64) red_add_release_gpu(comm.tile_done + (m_blk * TILE_M + (int)cta * CTA_M) / CTA_M, 1u);
      }
      if (++as == kAcc) { as = 0; aphase ^= 1; }
    }
    if constexpr (MODE == 2) {
      __threadfence();
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (threadIdx.x == 64) red_add_release_gpu(comm.gemm_done, 1u);
    }
  }

  if constexpr (MODE == 2) {
    // ---- reducer: (own 128-row block, 256-column slab) items, all CTAs -------------------------------------------
    __syncthreads();
    const int slabs = (N + 255) / 256;
    const int items = blk128_per_rank * slabs;
    const uint32_t* myflags = (const uint32_t*)comm.peer_flags[comm.rank] + comm.flag_offset;
    const __nv_bfloat16* staging = (const __nv_bfloat16*)((const uint8_t*)comm.peer_bufs[comm.rank] + comm.buf_offset);
    const __nv_bfloat16* own = out + (size_t)comm.rank * comm.rows_per_rank * N;
    __nv_bfloat16* rout = (__nv_bfloat16*)comm.rs_out;
    bool own_ready = false;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
      const int mb = it / slabs, slab = it % slabs;
      if ((int)threadIdx.x < comm.world && (int)threadIdx.x != comm.rank)
        wait_flag_ge(myflags + threadIdx.x * kMaxRowBlocks + mb, comm.epoch);
      if (!own_ready && threadIdx.x == 0)
        while ((int32_t)(ld_acquire_gpu(comm.gemm_done) - comm.gemm_done_target) < 0) __nanosleep(128);
      own_ready = true;
      __syncthreads();
      const int c0 = slab * 256;
      const int cols = min(256, N - c0);
      const int vec_per_row = cols / 8;
      // 4 vectors per thread per iteration and two sources at a time → 8 independent 16-byte loads in flight
      constexpr int V = 4;
      const int total_vec = CTA_M * vec_per_row;
      const size_t src_stride = (size_t)comm.rows_per_rank * N;
      for (int base = threadIdx.x; base < total_vec; base += V * kThreads) {
        size_t off[V];
        bool ok[V];
        float acc[V][8];
#pragma unroll
        for (int u = 0; u < V; ++u) {
          const int idx = base + u * kThreads;
          ok[u] = idx < total_vec;
          const int r = ok[u] ? idx / vec_per_row : 0, v = ok[u] ? idx % vec_per_row : 0;
          off[u] = ((size_t)(mb * CTA_M + r)) * N + c0 + v * 8;
        }
#pragma unroll
        for (int u = 0; u < V; ++u) {
          const uint4 raw = ok[u] ? *(const uint4*)(own + off[u]) : make_uint4(0, 0, 0, 0);
          const __nv_bfloat162* h = (const __nv_bfloat162*)&raw;
#pragma unroll
          for (int j = 0; j < 4; ++j) { const float2 f = __bfloat1622float2(h[j]); acc[u][2 * j] = f.x; acc[u][2 * j + 1] = f.y; }
        }
        for (int s0 = 0; s0 < comm.world; s0 += 2) {
          uint4 raw[2][V];
#pragma unroll
          for (int d = 0; d < 2; ++d) {
            const int sidx = s0 + d;
            const bool use = sidx < comm.world && sidx != comm.rank;
#pragma unroll
            for (int u = 0; u < V; ++u)
              raw[d][u] = (use && ok[u]) ? *(const uint4*)(staging + (size_t)sidx * src_stride + off[u]) : make_uint4(0, 0, 0, 0);
          }
#pragma unroll
          for (int d = 0; d < 2; ++d)
#pragma unroll
            for (int u = 0; u < V; ++u) {
              const __nv_bfloat162* h = (const __nv_bfloat162*)&raw[d][u];
#pragma unroll
              for (int j = 0; j < 4; ++j) { const float2 f = __bfloat1622float2(h[j]); acc[u][2 * j] += f.x; acc[u][2 * j + 1] += f.y; }
            }
        }
#pragma unroll
        for (int u = 0; u < V; ++u) {
          if (!ok[u]) continue;
          uint4 o; __nv_bfloat162* oh = (__nv_bfloat162*)&o;
#pragma unroll
          for (int j = 0; j < 4; ++j) oh[j] = __floats2bfloat162_rn(acc[u][2 * j], acc[u][2 * j + 1]);
          *(uint4*)(rout + off[u]) = o;
        }
      }
      __syncthreads();
    }
  }

  tcgen05_fence_before();
  cluster_sync_all();
  if (warp == 1) { __syncwarp(); tcgen05_dealloc_2cta(tmem_base, kTmemCols); }
}

}  // namespace g2

// ------------------------------------------------------------------ host side
CUtensorMap make_tmap_bf16(const void* ptr, uint64_t rows, uint64_t cols, uint32_t box_cols, uint32_t box_rows);
int device_sm_count();

CUtensorMap make_tmap_mats(const void* ptr, bool f32, uint64_t mats, uint64_t rows, uint64_t cols, uint32_t box_cols, uint32_t box_rows);

template <bool AK, bool BK_, typename OutT, int MODE = 0, int TN = g2::TILE_N>
static void launch2(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& to, const CUtensorMap& tp, void* out, int M, int N, int K,
                    int accumulate, int split_k, const g2::Group& grp, const g2::Tail& tail, int grid, cudaStream_t st, const CUtensorMap* keep = nullptr) {
  auto kern = g2::gemm_bf16_2cta_kernel<AK, BK_, OutT, MODE, TN>;
  constexpr int smem = g2::Shape<TN>::kShared;
  NXD_ALLOW_SMEM(kern, smem);
  // A dependent: barriers, TMEM and maps of the next product are set up beside the end of this one (1 x 1000 tokens of 13B: 1152 us, 1130 with
  // products, their tails, norms, SwiGLU and rotation so).  Not the grouped ones: they read the blocks' experts first and gain nothing.
  if (g2::whole(MODE)) {
    launch_dependent(kern, grid, g2::kThreads, smem, st, ta, tb, to, tp, keep ? *keep : tp, (OutT*)out, M, N, K, accumulate, split_k, grp, tail);
  } else {
    kern<<<grid, g2::kThreads, smem, st>>>(ta, tb, to, tp, keep ? *keep : tp, (OutT*)out, M, N, K, accumulate, split_k, grp, tail);
    NXD_CUDA_CHECK(cudaGetLastError());
  }
}

// Map of an output: fp32 slabs of 32 columns, bf16 slabs of 64; bf16 outputs that accumulate take no map (a dummy).
static CUtensorMap out_map(const void* out, int out_dt, bool accumulate, bool mats, int groups, int M, int N, const CUtensorMap& dummy) {
  if (out_dt == kF32) return make_tmap_mats(out, true, groups, M, N, 32, g2::CTA_M);
  if (accumulate) return dummy;
  if (N % 8) nxd_throw("CTA-pair GEMM: bf16 output needs N % 8 == 0", __FILE__, __LINE__);
  return mats ? make_tmap_mats(out, false, groups, M, N, g2::kEpiSlabCols, g2::CTA_M) : make_tmap_bf16(out, M, N, g2::kEpiSlabCols, g2::CTA_M);
}

// How a product is shared out: tiles of 256 or 128 columns; split-K of every tile (fp32 outputs), or of the last round's tiles alone, or neither.
// In us, for the estimates: a k-block of a 256 x 256 tile and of one of 256 x 128 (their operands, 32 and 24 KB a CTA, come at about 105 GB/s an
// SM); the launch that sums a tail; a MB of a tail's fp32 parts and of a pass over fp32 outputs.
constexpr double kWideUs = 0.31, kNarrowUs = 0.2325, kTailUs = 2.0, kPartUs = 1 / 7.0, kPassUs = 1 / 6.0;
// A tail's parts fill at most this many rounds of pairs, 58 MB of fp32 on 148 SMs: what a product may take beside its output.  In one, two, three
// and any number of rounds, us: 2048 x 4096 x 22016 308 / 310 / 292 / 292 (57 MB), 2048 x 4096 x 32000 464 / 468 / 426 / 429 (57), 512 x 5120 x 27648
// 163 / 141 / 137 / 137 (52), 704 x 4096 x 22016 159 / 117 / 116 / 116 (38), 1000 x 4096 x 32064 216 in all.  Without it 134 MB for
// 1000 x 4096 x 128256.
constexpr int kTailRounds = 3;
struct GemmPlan { int tiles, split, width; g2::Tail tail; };      // width: columns of a tile
static GemmPlan gemm_plan(int M, int N, int K, int out_dt, bool accumulate, bool split_k, bool narrow = true) {
  const int pairs = std::max(1, device_sm_count() / 2), num_kb = (K + g2::BK - 1) / g2::BK;      // (no device: one, for the asking)
  const int tiles_m = (M + g2::TILE_M - 1) / g2::TILE_M;
  GemmPlan p;
  double best = 1e30;
  for (int width = 256; width >= (narrow ? 128 : 256); width /= 2) {
    const double kb_us = width == 256 ? kWideUs : kNarrowUs;
    const int tiles = tiles_m * ((N + width - 1) / width);
    // The tail: the tiles of the last, partial round in s parts each, which may be several rounds themselves; worth it where it saves more than
    // the launch that sums and its traffic.  Chosen so and before (256 columns, s pairs a tile in one round), us: 512 x 5120 x 13824 in 3
    // parts 64 and 74; 704 x 4096 x 11008 in 3 parts 56 and 62; 304 x 4096 x 4096 in 128 columns 19.6 and 21.2, 304 x 1024 x 2816 in 128 columns
    // and 4 parts 10.6 and 15.8, 1000 x 1024 x 1024 in 128 columns 8.2 and 10.0; 1000 x 5120 x 13824 (80 tiles) 101 in 5 parts, 147 without.  66
    // such products of 200 to 1504 rows: none slower than before by more than its noise but one (200 x 4096 x 11008, 37 and 34), a twelfth of a per
    // cent from the best of all these choices in the mean.
    // Rows of other lengths have no tail: gemm_tail_kernel writes whole groups of 8 columns.
    const int last = N % 8 == 0 ? tiles % pairs : 0;
    for (int s = 1; s <= (last > 0 ? 16 : 1); ++s) {
      const int per = (num_kb + s - 1) / s;
      if (s > 1 && (num_kb / s < 4 || per * (s - 1) >= num_kb)) continue;      // short parts, or an empty one
      if (s > 1 && last * s * width > kTailRounds * pairs * g2::TILE_N) break;
      const int rounds = (last * s + pairs - 1) / pairs;
      double cost = ((tiles / pairs) * num_kb + rounds * per) * kb_us + (s > 1 ? kTailUs + 2.0 * last * s * width * 0.001024 * kPartUs : 0.);
      if (s > 1) cost /= 0.97;                             // a tie stays whole
      if (cost < best) {
        best = cost;
        p.tiles = tiles; p.split = 1; p.width = width;
        p.tail = s > 1 ? g2::Tail{last, s, per} : g2::Tail{0, 1, num_kb};
      }
    }
  }
  // Split-K for fp32 outputs (weight gradients): K = tokens is long while the output often has fewer tiles than the
  // chip has CTA pairs (TP=8: 32-176 tiles on 74 pairs).  A split is taken where the waves it saves cost more than its traffic:
  // zeroing the output first and one more pass over it per further partial; every split keeps >= 16 k-blocks so that the main
  // loop still amortises its epilogue.  Its partials are added in any order.  Outputs of fewer rows than a tile never take it: their few
  // tiles are a tail, whose partials are summed in order, so that the same inputs give the same bits.
  if (out_dt == kF32 && M >= g2::TILE_M && split_k) {
    const int tiles = tiles_m * ((N + g2::TILE_N - 1) / g2::TILE_N);
    const double pass_us = (double)M * N * 4e-6 * kPassUs;
    for (int s2 = 2; s2 <= 8; ++s2) {
      if (num_kb / s2 < 16) break;
      const int per = (num_kb + s2 - 1) / s2;
      if (per * (s2 - 1) >= num_kb) continue;                       // would leave an empty split
      const double cost = (double)((tiles * s2 + pairs - 1) / pairs) * per * kWideUs + (s2 - 1) * pass_us + (accumulate ? 0. : pass_us);
      if (cost < best) {
        best = cost;
        p.tiles = tiles; p.split = s2; p.width = g2::TILE_N;
        p.tail = g2::Tail{0, 1, num_kb};
      }
    }
  }
  return p;
}

// bytes of fp32 workspace that gemm_bf16_2cta takes for these sizes (0: none; at most kTailRounds * 256 KB for each pair of SMs)
size_t gemm_2cta_workspace(int M, int N, int K, int out_dt, bool accumulate, bool split_k) {
  const GemmPlan p = gemm_plan(M, N, K, out_dt, accumulate, split_k);
  return (size_t)p.tail.tiles * p.tail.splits * g2::TILE_M * p.width * sizeof(float);
}

// `split_k`: fp32 outputs may be sums in any order; `workspace`: gemm_2cta_workspace bytes, 16-byte aligned, or null: then no tail is split
void gemm_bf16_2cta(const void* a, const void* b, void* out, int M, int N, int K, bool trans_a, bool trans_b, int out_dt,
                    bool accumulate, bool split_k, float* workspace, cudaStream_t st) {
  const bool AK = !trans_a, BK_ = trans_b;
  const CUtensorMap ta = AK ? make_tmap_bf16(a, M, K, g2::BK, g2::CTA_M) : make_tmap_bf16(a, K, M, 64, g2::BK);
  GemmPlan p = gemm_plan(M, N, K, out_dt, accumulate, split_k);
  const CUtensorMap tb = BK_ ? make_tmap_bf16(b, N, K, g2::BK, p.width / 2) : make_tmap_bf16(b, K, N, 64, g2::BK);
  const CUtensorMap to = out_map(out, out_dt, accumulate, false, 1, M, N, ta);
  if (!workspace) p.tail = g2::Tail{0, 1, 1};
  const int pairs = device_sm_count() / 2, split = p.split;
  if (split > 1 && !accumulate) NXD_CUDA_CHECK(cudaMemsetAsync(out, 0, (size_t)M * N * sizeof(float), st));   // partials add into zeros
  const CUtensorMap tp = p.tail.tiles ? make_tmap_mats(workspace, true, (uint64_t)p.tail.tiles * p.tail.splits, g2::TILE_M, p.width, 32, g2::CTA_M) : ta;
  const int units = p.tiles * split + p.tail.tiles * (p.tail.splits - 1);
  const int grid = 2 * (units < pairs ? units : pairs);
  const g2::Group none{};
#define NXD_L2W(AKv, BKv, OutT, W) launch2<AKv, BKv, OutT, 0, W>(ta, tb, to, tp, out, M, N, K, accumulate, split, none, p.tail, grid, st)
#define NXD_L2(AKv, BKv)                                                                                              \
  do {                                                                                                                \
    if (out_dt == kBF16) { if (p.width == 128) NXD_L2W(AKv, BKv, __nv_bfloat16, 128); else NXD_L2W(AKv, BKv, __nv_bfloat16, 256); } \
    else { if (p.width == 128) NXD_L2W(AKv, BKv, float, 128); else NXD_L2W(AKv, BKv, float, 256); }                    \
  } while (0)
  if (AK && BK_) NXD_L2(true, true);
  else if (AK && !BK_) NXD_L2(true, false);
  else if (!AK && !BK_) NXD_L2(false, false);
  else NXD_L2(false, true);
#undef NXD_L2
#undef NXD_L2W
  if (p.tail.tiles) {
    const int tiles_m = (M + g2::TILE_M - 1) / g2::TILE_M, tiles_n = (N + p.width - 1) / p.width;
    const dim3 tg(g2::TILE_M * p.width / 2048, p.tail.tiles);
    auto sum = [&](auto kernel, auto* o) {
      launch_dependent(kernel, tg, 256, 0, st, (const float*)workspace, o, M, N, p.tiles - p.tail.tiles, tiles_m, tiles_n, p.tail.splits, (int)accumulate, decltype(o)(nullptr));
    };
    if (out_dt == kBF16) sum(p.width == 128 ? g2::gemm_tail_kernel<__nv_bfloat16, 128> : g2::gemm_tail_kernel<__nv_bfloat16, 256>, (__nv_bfloat16*)out);
    else sum(p.width == 128 ? g2::gemm_tail_kernel<float, 128> : g2::gemm_tail_kernel<float, 256>, (float*)out);
    NXD_CUDA_CHECK(cudaGetLastError());
  }
}

// y [M, I] = SwiGLU of x [M, K] · w [2 I, K]ᵀ (gate rows first), I a multiple of 128: the products stay in tensor memory instead of going to memory
// and through another kernel; with `keep` they go to [M, 2 I] as well, and what is saved is reading them again.  The same bits as the two kernels
// where the tiles are the same.
size_t gemm_swiglu_2cta_workspace(int M, int I, int K) {
  const GemmPlan p = gemm_plan(M, 2 * I, K, kBF16, false, false, false);
  return (size_t)p.tail.tiles * p.tail.splits * g2::TILE_M * p.width * sizeof(float);
}
void gemm_swiglu_2cta(const void* x, const void* w, void* y, void* keep, int M, int I, int K, float* workspace, cudaStream_t st) {
  if (I % 128 || K % 8) nxd_throw("gemm_swiglu_2cta: I must be a multiple of 128, K of 8", __FILE__, __LINE__);
  const CUtensorMap ta = make_tmap_bf16(x, M, K, g2::BK, g2::CTA_M), tb = make_tmap_bf16(w, 2l * I, K, g2::BK, g2::HALF_N);
  const CUtensorMap to = make_tmap_bf16(y, M, I, g2::kEpiSlabCols, g2::CTA_M);
  GemmPlan p = gemm_plan(M, 2 * I, K, kBF16, false, false, false);
  if (!workspace) p.tail = g2::Tail{0, 1, 1};
  const int pairs = device_sm_count() / 2, units = p.tiles + p.tail.tiles * (p.tail.splits - 1), grid = 2 * (units < pairs ? units : pairs);
  const CUtensorMap tp = p.tail.tiles ? make_tmap_mats(workspace, true, (uint64_t)p.tail.tiles * p.tail.splits, g2::TILE_M, p.width, 32, g2::CTA_M) : ta;
  if (keep) {
    const CUtensorMap tk = make_tmap_bf16(keep, M, 2l * I, g2::kEpiSlabCols, g2::CTA_M);
    launch2<true, true, __nv_bfloat16, 6>(ta, tb, to, tp, y, M, I, K, 0, 1, g2::Group{}, p.tail, grid, st, &tk);
  } else {
    launch2<true, true, __nv_bfloat16, 5>(ta, tb, to, tp, y, M, I, K, 0, 1, g2::Group{}, p.tail, grid, st);
  }
  if (p.tail.tiles)
    launch_dependent(g2::gemm_tail_kernel<__nv_bfloat16, 256, true>, dim3(g2::TILE_M / 16, p.tail.tiles), 256, 0, st, (const float*)workspace, (__nv_bfloat16*)y,
                     M, I, p.tiles - p.tail.tiles, (M + g2::TILE_M - 1) / g2::TILE_M, I / 128, p.tail.splits, 0, (__nv_bfloat16*)keep);
  NXD_CUDA_CHECK(cudaGetLastError());
}

// Grouped GEMMs of routed experts whose row blocks are multiples of 256 rows (see grouped_gemm_bf16 / grouped_wgrad_bf16).
void grouped_gemm_bf16_2cta(const void* a, const void* b, void* out, int M, int N, int K, int E, bool trans_b, const int* block_expert,
                            const int* used_blocks, int block_rows, int out_dt, cudaStream_t st) {
  const CUtensorMap ta = make_tmap_bf16(a, M, K, g2::BK, g2::CTA_M);
  const CUtensorMap tb = trans_b ? make_tmap_bf16(b, (uint64_t)E * N, K, g2::BK, g2::HALF_N) : make_tmap_bf16(b, (uint64_t)E * K, N, 64, g2::BK);
  const CUtensorMap to = out_map(out, out_dt, false, false, 1, M, N, ta);
  const g2::Group grp{block_expert, nullptr, used_blocks, block_rows, trans_b ? N : K, E, nullptr};
  const int tiles = ((M + g2::TILE_M - 1) / g2::TILE_M) * ((N + g2::TILE_N - 1) / g2::TILE_N), pairs = device_sm_count() / 2;
  const int grid = 2 * (tiles < pairs ? tiles : pairs);
  if (trans_b) {
    if (out_dt == kBF16) launch2<true, true, __nv_bfloat16, 3>(ta, tb, to, to, out, M, N, K, 0, 1, grp, g2::Tail{0, 1, 1}, grid, st);
    else launch2<true, true, float, 3>(ta, tb, to, to, out, M, N, K, 0, 1, grp, g2::Tail{0, 1, 1}, grid, st);
  } else {
    if (out_dt == kBF16) launch2<true, false, __nv_bfloat16, 3>(ta, tb, to, to, out, M, N, K, 0, 1, grp, g2::Tail{0, 1, 1}, grid, st);
    else launch2<true, false, float, 3>(ta, tb, to, to, out, M, N, K, 0, 1, grp, g2::Tail{0, 1, 1}, grid, st);
  }
}

// y [M, I] = SwiGLU of the routed rows' products with their expert's [K, gate up] weights b [E, K, 2 I], I a multiple of 128; keep, if any: the products
void grouped_swiglu_2cta(const void* a, const void* b, void* y, void* keep, int M, int I, int K, int E, const int* block_expert, const int* used_blocks,
                         int block_rows, cudaStream_t st) {
  if (I % 128 || K % 64 || block_rows % g2::TILE_M) nxd_throw("grouped_swiglu_2cta: I in 128s, K in 64s, blocks of 256 rows", __FILE__, __LINE__);
  const CUtensorMap ta = make_tmap_bf16(a, M, K, g2::BK, g2::CTA_M), tb = make_tmap_bf16(b, (uint64_t)E * K, 2l * I, 64, g2::BK);
  const CUtensorMap to = make_tmap_bf16(y, M, I, g2::kEpiSlabCols, g2::CTA_M);
  const CUtensorMap tk = keep ? make_tmap_bf16(keep, M, 2l * I, g2::kEpiSlabCols, g2::CTA_M) : to;
  const g2::Group grp{block_expert, nullptr, used_blocks, block_rows, K, E, nullptr};
  const int tiles = ((M + g2::TILE_M - 1) / g2::TILE_M) * (I / 128), pairs = device_sm_count() / 2, grid = 2 * (tiles < pairs ? tiles : pairs);
  launch2<true, false, __nv_bfloat16, 7>(ta, tb, to, to, y, M, I, K, keep != nullptr, 1, grp, g2::Tail{0, 1, 1}, grid, st, &tk);
}

void grouped_wgrad_bf16_2cta(const void* a, const void* b, void* out, int rows_total, int Mo, int No, int E, const int* seg_first_block,
                             const int* slot_token, int block_rows, int out_dt, bool accumulate, cudaStream_t st) {
  const CUtensorMap ta = make_tmap_bf16(a, rows_total, Mo, 64, g2::BK);
  const CUtensorMap tb = make_tmap_bf16(b, rows_total, No, 64, g2::BK);
  const CUtensorMap to = out_map(out, out_dt, accumulate, true, E, Mo, No, ta);
  const g2::Group grp{nullptr, seg_first_block, nullptr, block_rows, 0, E, slot_token};
  const int tiles = E * ((Mo + g2::TILE_M - 1) / g2::TILE_M) * ((No + g2::TILE_N - 1) / g2::TILE_N), pairs = device_sm_count() / 2;
  const int grid = 2 * (tiles < pairs ? tiles : pairs);
  if (out_dt == kBF16) launch2<false, false, __nv_bfloat16, 4>(ta, tb, to, to, out, Mo, No, rows_total, accumulate, 1, grp, g2::Tail{0, 1, 1}, grid, st);
  else launch2<false, false, float, 4>(ta, tb, to, to, out, Mo, No, rows_total, accumulate, 1, grp, g2::Tail{0, 1, 1}, grid, st);
}


template <bool AK, bool BK_, int MODE>
static void launch_tp(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tal, void* out, int M, int N, int K,
                      const g2::TpComm& c, int grid, cudaStream_t st) {
  auto kern = g2::gemm_bf16_2cta_tp_kernel<AK, BK_, MODE>;
  NXD_ALLOW_SMEM(kern, g2::kSmem);
  kern<<<grid, g2::kThreads, g2::kSmem, st>>>(ta, tb, tal, (__nv_bfloat16*)out, M, N, K, c);
  NXD_CUDA_CHECK(cudaGetLastError());
}

// mode 1: `a` = this rank's gathered buffer [M,K] inside the symmetric payload, `a_local` = shard; out = [M,N].
// mode 2: `a` = [M,K]; `partial` = local [M,N] scratch; `rs_out` = [M/world, N].
void gemm_bf16_2cta_tp(int mode, const void* a, const void* b, void* out_or_partial, void* rs_out, const void* a_local,
                       int M, int N, int K, bool trans_b, int rank, int world, const int64_t* peer_bufs,
                       const int64_t* peer_flags, long buf_offset, int flag_offset, uint32_t epoch, int comm_ctas,
                       uint32_t* tile_done, uint32_t* gemm_done, uint32_t gemm_done_target, cudaStream_t st) {
  const bool BK_ = trans_b;
  const CUtensorMap ta = make_tmap_bf16(a, M, K, g2::BK, g2::CTA_M);
  const CUtensorMap tb = BK_ ? make_tmap_bf16(b, N, K, g2::BK, g2::HALF_N) : make_tmap_bf16(b, K, N, 64, g2::BK);
  g2::TpComm c{};
  c.mode = mode; c.rank = rank; c.world = world; c.peer_bufs = peer_bufs; c.peer_flags = peer_flags;
  c.buf_offset = buf_offset; c.flag_offset = flag_offset; c.epoch = epoch; c.comm_ctas = comm_ctas;
  c.rows_per_rank = M / world; c.a_local = a_local; c.rs_out = rs_out; c.tile_done = tile_done; c.gemm_done = gemm_done;
  c.gemm_done_target = gemm_done_target;
  { const char* e = getenv("NXD_TP_PUSH");      // re-read per call (sweeps): ldst | tma (default) | stream (opt-in, see tma_push_stream)
    c.push_tma = !e ? 1 : (std::string(e) == "ldst" ? 0 : (std::string(e) == "stream" ? 2 : 1)); }
  if (M % world || c.rows_per_rank % g2::TILE_M || c.rows_per_rank / g2::CTA_M > g2::kMaxRowBlocks)
    nxd_throw("fused TP GEMM (CTA-pair) needs rows/rank to be a multiple of 256 and <= 8192", __FILE__, __LINE__);
  const int grid = (device_sm_count() / 2) * 2;
  const CUtensorMap tal = (mode == 1) ? make_tmap_bf16(a_local, c.rows_per_rank, K, g2::BK, g2::CTA_M) : ta;
  if (mode == 1) { if (BK_) launch_tp<true, true, 1>(ta, tb, tal, out_or_partial, M, N, K, c, grid, st);
                   else launch_tp<true, false, 1>(ta, tb, tal, out_or_partial, M, N, K, c, grid, st); }
  else { if (BK_) launch_tp<true, true, 2>(ta, tb, tal, out_or_partial, M, N, K, c, grid, st);
         else launch_tp<true, false, 2>(ta, tb, tal, out_or_partial, M, N, K, c, grid, st); }
}

}  // namespace nxd

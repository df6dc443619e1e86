// Shared pieces of the CTA-pair (cta_group::2) bf16 GEMM kernels: tile constants, the TMEM→global epilogue store and the
// 256-row raster.  Included by gemm2cta_sm100.cu (plain + unicast TP kernels) and tp_nvls_sm100.cu (NVLS TP kernels).
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace nxd {
namespace g2 {

constexpr int TILE_M = 256;         // per pair
constexpr int CTA_M = 128;
constexpr int TILE_N = 256;
constexpr int HALF_N = 128;         // B rows staged per CTA
constexpr int BK = 64;
constexpr int UK = 16;
constexpr int kStages = 6;
constexpr int kAcc = 2;
constexpr int kABytes = CTA_M * BK * 2;      // 16 KB
constexpr int kBBytes = HALF_N * BK * 2;     // 16 KB
constexpr int kStageBytes = kABytes + kBBytes;
constexpr int kThreads = 192;
// epilogue staging: two 128-row x 64-column bf16 slabs (128B-swizzled rows), written by the epilogue warps and drained by
// TMA bulk tensor stores — coalesced, asynchronous, no per-thread row-strided global stores
constexpr int kEpiSlabCols = 64;
constexpr int kEpiSlabBytes = CTA_M * kEpiSlabCols * 2;   // 16 KB
constexpr int kEpiBufs = 2;
constexpr int kEpiOffset = kStages * kStageBytes;
constexpr int kBarOffset = kEpiOffset + kEpiBufs * kEpiSlabBytes;
constexpr int kSmem = kBarOffset + 1024 + 256;
constexpr int kTmemCols = kAcc * TILE_N;     // 512
static_assert(kSmem <= 232448, "exceeds the 227 KB of dynamic shared memory per CTA");

template <typename OutT>
NXD_DEVICE void store_chunk(OutT* orow, int col0, int N, const uint32_t (&r)[32], int accumulate) {
  if constexpr (sizeof(OutT) == 2) {
    if (col0 + 32 <= N) {
      uint4 pk[4];
      __nv_bfloat162* h = (__nv_bfloat162*)pk;
      if (accumulate) {
        const uint4* old = (const uint4*)(orow + col0);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const uint4 o = old[v];
          const __nv_bfloat162* oh = (const __nv_bfloat162*)&o;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 of = __bfloat1622float2(oh[j]);
            h[v * 4 + j] = __floats2bfloat162_rn(__uint_as_float(r[v * 8 + 2 * j]) + of.x,
                                                 __uint_as_float(r[v * 8 + 2 * j + 1]) + of.y);
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) h[j] = __floats2bfloat162_rn(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
      }
      uint4* dst = (uint4*)(orow + col0);
#pragma unroll
      for (int v = 0; v < 4; ++v) dst[v] = pk[v];
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        if (col0 + j < N) {
          float v = __uint_as_float(r[j]);
          if (accumulate) v += __bfloat162float(((__nv_bfloat16*)orow)[col0 + j]);
          ((__nv_bfloat16*)orow)[col0 + j] = __float2bfloat16_rn(v);
        }
      }
    }
  } else {
    if (col0 + 32 <= N) {                    // fp32 outputs that accumulate leave through epilogue_tile_tma_f32
      float4* dst = (float4*)(orow + col0);
#pragma unroll
      for (int v = 0; v < 8; ++v)
        dst[v] = make_float4(__uint_as_float(r[4 * v]), __uint_as_float(r[4 * v + 1]), __uint_as_float(r[4 * v + 2]),
                             __uint_as_float(r[4 * v + 3]));
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (col0 + j < N) ((float*)orow)[col0 + j] = __uint_as_float(r[j]);
    }
  }
}

// The four products of a k-block and the commit that frees its stage in both CTAs, from a warp that is together: one election, descriptors that
// advance by constants (steps of 16 bytes).  One lane on its own took about 130 cycles a product, as long as one of 256 columns lasts and
// twice as long as one of 128.
template <int STEP_A, int STEP_B>
NXD_DEVICE void mma4_commit_2cta(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred p, q, t;\n\t.reg .b64 a, b;\n\t"
      "elect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "add.s64 a, %1, %6;\n\tadd.s64 b, %2, %9;\n\t@q tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, t;\n\t"
      "add.s64 a, %1, %7;\n\tadd.s64 b, %2, %10;\n\t@q tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, t;\n\t"
      "add.s64 a, %1, %8;\n\tadd.s64 b, %2, %11;\n\t@q tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, t;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%5], %12;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(bar), "n"(STEP_A), "n"(2 * STEP_A), "n"(3 * STEP_A), "n"(STEP_B), "n"(2 * STEP_B),
        "n"(3 * STEP_B), "h"((uint16_t)3)
      : "memory");
}

// Row tiles that go through the columns together.  What the 74 tiles in flight share is read from memory once for each such pass over the columns:
// all row tiles at once where they are few, so that a large B is read once, near-square rounds (8 x 9 tiles) else.  Training products run under
// the power cap, where bytes cost time: feed-forward block of 7B, 4096 tokens, both ways, 2731 us with four rows, 2670 so.
NXD_DEVICE int raster_rows(int tiles_m) { return tiles_m <= 16 ? 16 : 8; }
NXD_DEVICE void tile_coords(int tile, int tiles_m, int tiles_n, int group, int& m_blk, int& n_blk) {
  const int per_group = group * tiles_n;
  const int g = tile / per_group;
  const int first_m = g * group;
  const int gsz = min(group, tiles_m - first_m);
  const int in = tile - g * per_group;
  m_blk = first_m + in % gsz;
  n_blk = in / gsz;
}


NXD_DEVICE void tma_store_2d(const CUtensorMap* map, uint32_t smem_src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(map), "r"(smem_src), "r"(c0), "r"(c1) : "memory");
}
NXD_DEVICE void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N_> NXD_DEVICE void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N_) : "memory"); }
template <int N_> NXD_DEVICE void bulk_wait() { asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N_) : "memory"); }
NXD_DEVICE void bulk_wait_n(int n) {       // all but the newest n bulk groups have fully completed (n in 0..4)
  switch (n) {
    case 0: bulk_wait<0>(); break;
    case 1: bulk_wait<1>(); break;
    case 2: bulk_wait<2>(); break;
    case 3: bulk_wait<3>(); break;
    default: bulk_wait<4>(); break;
  }
}

NXD_DEVICE void tma_store_3d(const CUtensorMap* map, uint32_t smem_src, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(map), "r"(smem_src), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
NXD_DEVICE void tma_reduce_add_3d(const CUtensorMap* map, uint32_t smem_src, int c0, int c1, int c2) {
  asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(map), "r"(smem_src), "r"(c0), "r"(c1), "r"(c2) : "memory");
}

// fp32 twin of epilogue_tile_tma below: slabs of 32 columns (128-byte rows again) leave through a 3-D map {columns, rows, matrices},
// as a plain store or added to memory by the copy engine (`add`: gradient accumulation, split-K partials).  A weight gradient is
// bound by these writes as much as by its products: with one row-strided 16-byte store per thread and instruction the tensor pipe
// waited for the epilogue.  7B feed-forward weight gradients over 4096 tokens: 846 + 39 us (stores, zeroing for a split) -> 744.
template <int TN = TILE_N>          // columns of the tile
NXD_DEVICE void epilogue_tile_tma_f32(uint32_t tmem_acc, uint32_t stage_smem, const CUtensorMap* omap, int row0, int mat, int col0,
                                      int N, int q, int lane, bool issuer, uint32_t& slab_ctr, bool add, bool zero) {
  const int row = q * 32 + lane;
#pragma unroll 1
  for (int s = 0; s < TN / 32; ++s) {
    const int c0 = col0 + s * 32;
    if (c0 >= N) break;
    const uint32_t buf = stage_smem + (slab_ctr & 1u) * kEpiSlabBytes;
    uint32_t r[32];
    tcgen05_ld_32x32(tmem_acc + s * 32, r);
    if (issuer) bulk_wait_read<1>();
    asm volatile("bar.sync 1, 128;" ::: "memory");
    tcgen05_wait_ld();
    if (zero) {
#pragma unroll
      for (int j = 0; j < 32; ++j) r[j] = 0u;
    }
    const uint32_t rbase = buf + (uint32_t)row * 128u;
    const uint32_t sw = (uint32_t)(row & 7);
#pragma unroll
    for (int c = 0; c < 8; ++c)
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};"
                   ::"r"(rbase + (((uint32_t)c ^ sw) << 4)), "r"(r[4 * c]), "r"(r[4 * c + 1]), "r"(r[4 * c + 2]), "r"(r[4 * c + 3])
                   : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (issuer) {
      if (add) tma_reduce_add_3d(omap, buf, c0, row0, mat);
      else tma_store_3d(omap, buf, c0, row0, mat);
      bulk_commit();
    }
    ++slab_ctr;
  }
}

// Epilogue of one 128x256 accumulator (this CTA's TMEM lanes) to a row-major bf16 matrix through TMA stores.
// Executed by the 128 epilogue threads (warps 2-5, named barrier 1); thread `issuer` (one of them) owns the bulk groups.
// Per 64-column slab: wait until the staging buffer's previous store has read it, tcgen05.ld 2x32 columns, pack to bf16,
// write the thread's 128-byte row in the 128B-swizzle pattern (conflict-free: 8 consecutive rows hit 8 different 16-byte
// bank groups), fence to the async proxy, TMA-store the slab.  Rows/columns beyond the matrix are clipped by TMA.
// Returns the number of bulk groups committed (slabs inside the matrix).  `slab_ctr` carries the buffer parity.
template <bool MATS = false, int TN = TILE_N>      // MATS: a 3-D map {columns, rows, matrices}, matrix `mat`; `zero`: the accumulator was never written
NXD_DEVICE int epilogue_tile_tma(uint32_t tmem_acc, uint32_t stage_smem, const CUtensorMap* omap, int row0, int col0, int N,
                                 int q, int lane, bool issuer, uint32_t& slab_ctr, int mat = 0, bool zero = false) {
  const int row = q * 32 + lane;
  int groups = 0;
#pragma unroll 1
  for (int s = 0; s < TN / kEpiSlabCols; ++s) {
    const int c0 = col0 + s * kEpiSlabCols;
    if (c0 >= N) break;
    const uint32_t buf = stage_smem + (slab_ctr & 1u) * kEpiSlabBytes;
    if (issuer) bulk_wait_read<1>();
    asm volatile("bar.sync 1, 128;" ::: "memory");
    uint32_t r0[32], r1[32];
    tcgen05_ld_32x32(tmem_acc + s * kEpiSlabCols, r0);
    tcgen05_ld_32x32(tmem_acc + s * kEpiSlabCols + 32, r1);
    tcgen05_wait_ld();
    if constexpr (MATS) {
      if (zero) {
#pragma unroll
        for (int j = 0; j < 32; ++j) r0[j] = r1[j] = 0u;
      }
    }
    const uint32_t rbase = buf + (uint32_t)row * 128u;
    const uint32_t sw = (uint32_t)(row & 7);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const uint32_t* src = (c < 4) ? (r0 + 8 * c) : (r1 + 8 * (c - 4));
      uint4 pk;
      __nv_bfloat162* h = (__nv_bfloat162*)&pk;
#pragma unroll
      for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(__uint_as_float(src[2 * j]), __uint_as_float(src[2 * j + 1]));
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};"
                   ::"r"(rbase + (((uint32_t)c ^ sw) << 4)), "r"(pk.x), "r"(pk.y), "r"(pk.z), "r"(pk.w) : "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (issuer) {
      if constexpr (MATS) tma_store_3d(omap, buf, c0, row0, mat);
      else tma_store_2d(omap, buf, c0, row0);
      bulk_commit();
    }
    ++slab_ctr;
    ++groups;
  }
  return groups;
}

// The same for tiles whose first 128 columns are gates and last 128 ups: SwiGLU of the two, 128 columns from col0 on.
NXD_DEVICE void epilogue_tile_swiglu(uint32_t tmem_acc, uint32_t stage_smem, const CUtensorMap* omap, int row0, int col0, int q, int lane, bool issuer,
                                     uint32_t& slab_ctr) {
  const int row = q * 32 + lane;
#pragma unroll 1
  for (int s = 0; s < 2; ++s) {
    const uint32_t buf = stage_smem + (slab_ctr & 1u) * kEpiSlabBytes;
    if (issuer) bulk_wait_read<1>();
    asm volatile("bar.sync 1, 128;" ::: "memory");
    const uint32_t rbase = buf + (uint32_t)row * 128u;
    const uint32_t sw = (uint32_t)(row & 7);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t g[32], u[32];
      tcgen05_ld_32x32(tmem_acc + s * 64 + h * 32, g);
      tcgen05_ld_32x32(tmem_acc + 128 + s * 64 + h * 32, u);
      tcgen05_wait_ld();
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint4 pk;
        __nv_bfloat162* o = (__nv_bfloat162*)&pk;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int i = 8 * c + 2 * j;
          o[j] = __floats2bfloat162_rn(silu_mul_bf16(__uint_as_float(g[i]), __uint_as_float(u[i])),
                                       silu_mul_bf16(__uint_as_float(g[i + 1]), __uint_as_float(u[i + 1])));
        }
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};"
                     ::"r"(rbase + (((uint32_t)(h * 4 + c) ^ sw) << 4)), "r"(pk.x), "r"(pk.y), "r"(pk.z), "r"(pk.w) : "memory");
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (issuer) {
      tma_store_2d(omap, buf, col0 + s * 64, row0);
      bulk_commit();
    }
    ++slab_ctr;
  }
}

NXD_DEVICE uint32_t ld_acquire_gpu(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
NXD_DEVICE void red_add_release_gpu(uint32_t* p, uint32_t v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
NXD_DEVICE uint32_t atom_add_acqrel_gpu(uint32_t* p, uint32_t v) {
  uint32_t old;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}

}  // namespace g2
}  // namespace nxd

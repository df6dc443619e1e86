// y[M, N] = x[M, K] · W[N, K]ᵀ (+ residual) for few rows (speculation windows, short prompts, small batches): bf16, fp32 sums.
//
// Bound by reading W once.  The operands change places: 128 rows of W are the M side of the tensor-core product and the tokens
// (padded to a multiple of 16) its N side, so that a block streams a [128, K] slab of W and nothing of the tile is padding but
// the tokens' remainder.  What keeps HBM busy is bytes in flight, not tiles per SM: two blocks share an SM (each a ring of
// 16 KB W tiles), and where N has too few slabs the K range of a slab is split over a cluster of 2, 4 or 8 blocks, whose fp32
// partials are summed through distributed shared memory in a fixed order: no workspace, no atomics, no second launch.
// 48 rows, 22016 x 4096: 36 us (27.6 to read W; 40 with 128 x 256 tiles), 4096 x 11008: 21 us (13.8; 69 with 16 tiles for 148 SMs),
// 4096 x 4096: 12.9 us (5.1; 30).
// Its blocks start beside the kernel before it and ask for their first weight tiles (to L2: whoever wrote them is waited for before they are
// read).  48 rows through gate and up, SwiGLU and down of 4096 x 11008: 66.3 us, 60.6 without the tiles ahead, 59.6 with; a token of
// 13B for 4 sequences 386, 366, 360.
#include <cuda.h>

#include "common.cuh"
#include "kernels.h"
#include "sm100_ptx.cuh"

namespace nxd {

CUtensorMap make_tmap_bf16(const void* ptr, uint64_t rows, uint64_t cols, uint32_t box_cols, uint32_t box_rows);
int device_sm_count();

namespace few {

constexpr int kSlab = 128;                       // rows of W per block
constexpr int BK = 64;
constexpr int kWBytes = kSlab * BK * 2;          // 16 KB
constexpr int kThreads = 128;
constexpr int kMaxStages = 8;
constexpr int kBarBytes = 256;
constexpr int kAhead = 6;                        // weight tiles of a block brought to L2 while the kernel before it still runs

NXD_DEVICE void prefetch_l2_tile(const CUtensorMap* map, int c0, int c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(map), "r"(c0), "r"(c1) : "memory");
}
NXD_DEVICE float2 ld_cluster_f2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}
NXD_DEVICE float2 ld_shared_f2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}
// the four products of a k-block and the commit that frees its stage, from a warp that is together (one election; descriptors advance by 32 bytes)
NXD_DEVICE void mma4_commit(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred p, q, t;\n\t.reg .b64 a, b;\n\t"
      "elect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "add.s64 a, %1, 2;\n\tadd.s64 b, %2, 2;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t"
      "add.s64 a, %1, 4;\n\tadd.s64 b, %2, 4;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t"
      "add.s64 a, %1, 6;\n\tadd.s64 b, %2, 6;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%5];\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(bar) : "memory");
}
NXD_DEVICE float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// grid: split blocks (one cluster) per slab.  TN: tokens padded to 16; stage = W tile + x tile [TN, 64].
// GATE: W holds N gate rows and then N up rows, a slab 64 of each, and y [M, N] is SwiGLU of the two products (no residual).
template <bool GATE>
__global__ void __launch_bounds__(kThreads)
gemm_few_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_x, const __nv_bfloat16* residual,
                __nv_bfloat16* y, int M, int N, int K, int TN, int stages, int tmem_cols, int split) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int stage_bytes = kWBytes + TN * BK * 2;
  const int ring_bytes = max(stages * stage_bytes, TN * kSlab * 4);
  const uint32_t bars = base + ring_bytes;
  const uint32_t bar_full = bars, bar_empty = bars + 8 * kMaxStages, bar_done = bars + 16 * kMaxStages, tmem_slot = bar_done + 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = split > 1 ? (int)cluster_ctarank() : 0;
  constexpr int kCols = GATE ? kSlab / 2 : kSlab;          // outputs of a slab
  const int n0 = (int)blockIdx.x / split * kCols;
  const int num_kb = (K + BK - 1) / BK, per = (num_kb + split - 1) / split;
  const int kb0 = rank * per, kb1 = min(num_kb, kb0 + per);       // the host leaves no rank without a k-block

  if (threadIdx.x == 0) {
    prefetch_tmap(&tma_w); prefetch_tmap(&tma_x);
    for (int kb = kb0; kb < min(kb1, kb0 + kAhead); ++kb) {
      prefetch_l2_tile(&tma_w, kb * BK, n0);
      if constexpr (GATE) prefetch_l2_tile(&tma_w, kb * BK, N + n0);
    }
    for (int i = 0; i < stages; ++i) { mbar_init(bar_full + 8 * i, 1); mbar_init(bar_empty + 8 * i, 1); }
    mbar_init(bar_done, 1);
    fence_barrier_init();
  }
  if (warp == 1) { tcgen05_alloc(tmem_slot, tmem_cols); tcgen05_relinquish(); }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot));
  pdl_trigger();                                           // behind the allocation (launch_dependent)
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      int st = 0; uint32_t ph = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        mbar_wait(bar_empty + 8 * st, ph ^ 1);
        mbar_expect_tx(bar_full + 8 * st, stage_bytes);
        const uint32_t sw = base + st * stage_bytes;
        tma_load_2d(sw, &tma_w, bar_full + 8 * st, kb * BK, n0);                   // box {64, rows of a slab}
        if constexpr (GATE) tma_load_2d(sw + kWBytes / 2, &tma_w, bar_full + 8 * st, kb * BK, N + n0);
        tma_load_2d(sw + kWBytes, &tma_x, bar_full + 8 * st, kb * BK, 0);
        if (++st == stages) { st = 0; ph ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t idesc = make_idesc(false, false, kSlab, TN);
    int st = 0; uint32_t ph = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      mbar_wait(bar_full + 8 * st, ph);
      tcgen05_fence_after();
      const uint32_t sw = base + st * stage_bytes;
      mma4_commit(tmem, make_smem_desc(sw, 16, 1024), make_smem_desc(sw + kWBytes, 16, 1024), idesc, kb > kb0 ? 1u : 0u, bar_empty + 8 * st);
      if (++st == stages) { st = 0; ph ^= 1; }
    }
    tcgen05_commit_e(bar_done);
    __syncwarp();
  }
  // ---- partial → shared memory as [token][128] fp32 over the ring (its last tile has been multiplied)
  mbar_wait(bar_done, 0);
  tcgen05_fence_after();
  for (int c = 0; c < TN; c += 16) {
    uint32_t r[16];
    tcgen05_ld_32x16(tmem + ((uint32_t)(warp * 32) << 16) + c, r);
    tcgen05_wait_ld();
#pragma unroll
    for (int j = 0; j < 16; ++j)
      asm volatile("st.shared.b32 [%0], %1;" ::"r"(base + ((c + j) * kSlab + warp * 32 + lane) * 4), "r"(r[j]) : "memory");
  }
  tcgen05_fence_before();
  if (split > 1) cluster_sync_all(); else __syncthreads();
  if (warp == 1) { tcgen05_fence_after(); tcgen05_dealloc(tmem, tmem_cols); }
  // ---- rank r sums and writes tokens r*4 + warp, + 4*split, ...: 256 contiguous bytes per warp (GATE: 128)
  if constexpr (GATE) {
    const int n = n0 + lane * 2;
    for (int t = rank * 4 + warp; t < M; t += 4 * split) {
      const uint32_t at = base + (t * kSlab + lane * 2) * 4;
      float2 g, u;
      for (int s = 0; s < split; ++s) {
        const uint32_t from = split > 1 ? mapa_shared(at, s) : at;
        const float2 a = split > 1 ? ld_cluster_f2(from) : ld_shared_f2(from), b = split > 1 ? ld_cluster_f2(from + 256) : ld_shared_f2(from + 256);
        g = s ? make_float2(g.x + a.x, g.y + a.y) : a;
        u = s ? make_float2(u.x + b.x, u.y + b.y) : b;
      }
      if (n < N) *reinterpret_cast<__nv_bfloat162*>(y + (long)t * N + n) = __floats2bfloat162_rn(silu_mul_bf16(g.x, u.x), silu_mul_bf16(g.y, u.y));
    }
    if (split > 1) cluster_sync_all();
    return;
  }
  const int n = n0 + lane * 4;
  for (int t = rank * 4 + warp; t < M; t += 4 * split) {
    const uint32_t at = base + (t * kSlab + lane * 4) * 4;
    float4 a;
    if (split == 1) {
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w) : "r"(at) : "memory");
    } else {
      a = ld_cluster_f4(mapa_shared(at, 0));
      for (int s = 1; s < split; ++s) {
        const float4 b = ld_cluster_f4(mapa_shared(at, s));
        a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
      }
    }
    if (n < N) {
      uint2 o;
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
      if (residual) {
        o = *reinterpret_cast<const uint2*>(residual + (long)t * N + n);
        const float2 r0 = __bfloat1622float2(h[0]), r1 = __bfloat1622float2(h[1]);
        a.x += r0.x; a.y += r0.y; a.z += r1.x; a.w += r1.y;
      }
      h[0] = __floats2bfloat162_rn(a.x, a.y);
      h[1] = __floats2bfloat162_rn(a.z, a.w);
      *reinterpret_cast<uint2*>(y + (long)t * N + n) = o;
    }
  }
  if (split > 1) cluster_sync_all();             // peers may still read this block's partial
}

}  // namespace few

// N: outputs; `gate`: SwiGLU of 2 N products
static void few_rows(const void* x, const void* w, const void* residual, void* y, int M, int N, int K, int split, bool gate, cudaStream_t st) {
  using namespace few;
  const int kCols = gate ? kSlab / 2 : kSlab;
  if (M < 1 || M > 256 || N % 8 || K % 8) nxd_throw("gemm_few_rows: 1 to 256 rows, N and K multiples of 8", __FILE__, __LINE__);
  const int TN = (M + 15) / 16 * 16, slabs = (N + kCols - 1) / kCols, num_kb = (K + BK - 1) / BK;
  if (split == 0) {
    // up to 128 rows (two blocks per SM): until every SM has a block; above (one per SM): while they still fit at once.
    // 4096 x 11008 (32 slabs), 48 rows, split 1 / 2 / 4 / 8: 52 / 30 / 21.4 / 21.2 us; 256 rows: 69 / 45 / 31 / 58 (two rounds of blocks).
    const int sms = device_sm_count();
    split = 1;
    while (split < 8 && num_kb / (2 * split) >= 4 && (TN <= 128 ? slabs * split < sms : 2 * slabs * split <= sms)) split *= 2;
  }
  while (split > 1 && (num_kb + split - 1) / split * (split - 1) >= num_kb) split /= 2;      // no rank without a k-block
  const int stage_bytes = kWBytes + TN * BK * 2;
  const int room = TN <= 128 ? 112 * 1024 : 224 * 1024;       // two blocks per SM while their rings stay deep enough
  int stages = (room - 1024 - kBarBytes) / stage_bytes;
  if (stages > kMaxStages) stages = kMaxStages;
  const int ring_bytes = stages * stage_bytes > TN * kSlab * 4 ? stages * stage_bytes : TN * kSlab * 4;
  const int smem = 1024 + kBarBytes + ring_bytes;
  int cols = 32;
  while (cols < TN) cols *= 2;
  const CUtensorMap tw = make_tmap_bf16(w, gate ? 2l * N : N, K, BK, kCols), tx = make_tmap_bf16(x, M, K, BK, TN);
  if (gate) NXD_ALLOW_SMEM(gemm_few_kernel<true>, 226 * 1024);
  else NXD_ALLOW_SMEM(gemm_few_kernel<false>, 226 * 1024);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(slabs * split); cfg.blockDim = dim3(kThreads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[2]{};
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split; attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = 2;
  NXD_CUDA_CHECK(cudaLaunchKernelEx(&cfg, gate ? gemm_few_kernel<true> : gemm_few_kernel<false>, tw, tx, (const __nv_bfloat16*)residual,
                                    (__nv_bfloat16*)y, M, N, K, TN, stages, cols, split));
}

// split = 0: by rule
void gemm_few_rows(const void* x, const void* w, const void* residual, void* y, int M, int N, int K, int split, cudaStream_t st) {
  few_rows(x, w, residual, y, M, N, K, split, false, st);
}
void gemm_few_rows_swiglu(const void* x, const void* w, void* y, int M, int I, int K, cudaStream_t st) {
  few_rows(x, w, nullptr, y, M, I, K, 0, true, st);
}

}  // namespace nxd

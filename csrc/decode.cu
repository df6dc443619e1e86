// Token-generation (decode) kernels for sm_100a — both are HBM-bandwidth problems, so they are plain CUDA tuned for wide
// coalesced loads rather than tensor-core kernels:
//   decode_attention : one query token per sequence against the KV cache (flash-decoding: split over the cache length,
//                      GQA group processed together so K/V are read once per kv head), + a combine pass over the splits.
//                      Role of the reference's token-generation attention (modules/attention, models' TKG path).
//   gemv_bf16        : y[M≤8, N] = x[M, K] · W[N, K]ᵀ (+ optional residual) for batch-1..8 decode; every weight byte is read once
//                      with 16-byte loads, fp32 accumulation.
#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace nxd {

namespace {

constexpr int HD = 128;
constexpr int kDecWarps = 4;
constexpr int kDecThreads = kDecWarps * 32;
constexpr int kDecRows = 16;                                 // cache rows of one tile of a warp
constexpr int kDecTileBytes = kDecRows * HD * 2;             // 4 KB of K, as much of V
constexpr int dec_smem_bytes(int stages) { return kDecWarps * stages * 2 * kDecTileBytes; }      // 64 KB: three blocks per SM; 96: two

NXD_DEVICE void cp_async16(uint32_t dst, const void* src, bool live) {    // not live: 16 zero bytes, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
NXD_DEVICE void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> NXD_DEVICE void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
NXD_DEVICE void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
NXD_DEVICE void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {   // rows 8..15 of A are zero
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %5}, {%7, %8}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1));
}

// One block per (key/value head, sequence, stretch of the cache); its G <= 8 query heads share every row that is read.
// Bound by HBM: 512 bytes per cache row and key/value head.  Each warp walks 16-row tiles of its own through its own ring of
// cp.async stages (no block barrier in the loop): two stages and three blocks per SM, so that starts and ends of blocks lie under the others' copies,
// or, where a launch has no more than that, three stages (decode_attention).  Scores come from mma.sync
// (a 16 x 8 x 16 step holds all heads of the group; exact products, fp32 sums), so a row costs a few instructions per warp
// instead of a dot product with four shuffles per head; probabilities stay fp32 and meet V in fp32 FMAs, lane = 4 columns.
// With the merge, us, three stages and two: 8 sequences, 8192-row caches (three quarters in use), 32 heads on 8: 44.6 and 42.5; 16, 4096, 64 on 8:
// 55.6 and 50.6; 1, 8192, 64 on 8 (256 blocks): 14.3 and 16.7; 3, 300, 40 (240 blocks): 6.8 and 7.3; 1, 2048, 40 (320 blocks): 11.2 and 9.3 out of
// L2, but a 13B model's token, whose caches come from memory, 304 and 317.
template <int G, int kDecStages>
__global__ void __launch_bounds__(kDecThreads, kDecStages == 2 ? 3 : 2) decode_attn_kernel(
    const __nv_bfloat16* q, const __nv_bfloat16* kc, const __nv_bfloat16* vc,
    const long* positions, float* part_o, float* part_ml,
    __nv_bfloat16* out, int B, int H, int Hkv, int L,
    long k_sb, long k_ss, long k_sh, long v_sb, long v_ss, long v_sh, long q_sb, long q_sh, long o_sb, long o_sh,
    float scale_log2, int splits) {
  extern __shared__ __align__(128) uint8_t dec_smem[];
  const int kvh = blockIdx.x, b = blockIdx.y, split = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_trigger();                                           // the merge's blocks may take their places; they wait for this grid
  pdl_wait();
  const long pos = positions[b];
  const int n_valid = (int)(pos < 0 ? 0 : (pos >= L ? L : pos + 1));
  const int per = (n_valid + splits - 1) / splits;
  const int s0 = split * per, s1 = min(n_valid, s0 + per);
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(dec_smem) + warp * (kDecStages * 2 * kDecTileBytes);
  const __nv_bfloat16* kb = kc + b * k_sb + (long)kvh * k_sh;
  const __nv_bfloat16* vb = vc + b * v_sb + (long)kvh * v_sh;

  // 16 lanes copy one 256-byte row, 16-byte chunk c of row r lands at chunk (c ^ (r & 7)): both ways of reading are conflict-free
  const int cr = lane >> 4, cc = lane & 15;
  auto load_tile = [&](int row0, int stage) {
    const uint32_t dst = ring + stage * (2 * kDecTileBytes);
#pragma unroll
    for (int i = 0; i < kDecRows / 2; ++i) {
      const int r = i * 2 + cr, s = row0 + r;
      const bool live = s < s1;
      const long at = live ? s : s0;                       // a row that exists, read or not
      const uint32_t off = r * 256 + ((cc ^ (r & 7)) << 4);
      cp_async16(dst + off, kb + at * k_ss + cc * 8, live);
      cp_async16(dst + kDecTileBytes + off, vb + at * v_ss + cc * 8, live);
    }
  };
  const int first = s0 + warp * kDecRows;
  const int tiles = first < s1 ? (s1 - first + kDecWarps * kDecRows - 1) / (kDecWarps * kDecRows) : 0;
#pragma unroll
  for (int st = 0; st < kDecStages - 1; ++st) {
    if (st < tiles) load_tile(first + st * kDecWarps * kDecRows, st);
    cp_async_commit();
  }

  // query fragments: row = head of the group (rows >= G zero), two 32-bit words per 16 columns
  const int hq = lane >> 2, quad = lane & 3;
  uint32_t qa[8][2];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    qa[k][0] = qa[k][1] = 0u;
    if (hq < G) {
      const __nv_bfloat16* qp = q + b * q_sb + (long)(kvh * G + hq) * q_sh + k * 16 + quad * 2;
      qa[k][0] = *reinterpret_cast<const uint32_t*>(qp);
      qa[k][1] = *reinterpret_cast<const uint32_t*>(qp + 8);
    }
  }
  __shared__ __align__(16) float sm_p[kDecWarps][kDecRows][G];
  float m = -INFINITY, l = 0.f;                            // of head hq; l of this lane's columns only
  float o[G][4];
#pragma unroll
  for (int g = 0; g < G; ++g)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[g][i] = 0.f;

  for (int t = 0; t < tiles; ++t) {
    const int row0 = first + t * kDecWarps * kDecRows;
    cp_async_wait<kDecStages - 2>();
    __syncwarp();                                          // tile t of all lanes is there; all lanes are done with tile t - 1
    if (t + kDecStages - 1 < tiles) load_tile(row0 + (kDecStages - 1) * kDecWarps * kDecRows, (t + kDecStages - 1) % kDecStages);
    cp_async_commit();
    const uint32_t ks = ring + (t % kDecStages) * (2 * kDecTileBytes), vs = ks + kDecTileBytes;
    float d[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      // matrices: rows 0-7 / columns 16k.., rows 0-7 / 16k + 8.., rows 8-15 / 16k.., rows 8-15 / 16k + 8..
      const int r = ((lane >> 4) << 3) + (lane & 7), c = k * 2 + ((lane >> 3) & 1);
      uint32_t kf[4];
      ldmatrix_x4(kf, ks + r * 256 + ((c ^ (r & 7)) << 4));
      mma_bf16(d[0], qa[k][0], qa[k][1], kf[0], kf[1]);
      mma_bf16(d[1], qa[k][0], qa[k][1], kf[2], kf[3]);
    }
    float sc[4] = {d[0][0] * scale_log2, d[0][1] * scale_log2, d[1][0] * scale_log2, d[1][1] * scale_log2};
    if (row0 + kDecRows > s1) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (row0 + (i >> 1) * 8 + quad * 2 + (i & 1) >= s1) sc[i] = -INFINITY;
    }
    float mx = fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const bool grew = mx > m;
    if (__any_sync(0xffffffffu, grew)) {
      const float mn = fmaxf(m, mx);
      const float corr = grew ? exp2f(m - mn) : 1.f;       // m = -inf: 0
      m = mn;
      l *= corr;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float c = __shfl_sync(0xffffffffu, corr, g * 4);
#pragma unroll
        for (int i = 0; i < 4; ++i) o[g][i] *= c;
      }
    }
    const float ms = m == -INFINITY ? 0.f : m;
    float p[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) { p[i] = exp2f(sc[i] - ms); l += p[i]; }
    if (hq < G) {
#pragma unroll
      for (int i = 0; i < 4; ++i) sm_p[warp][(i >> 1) * 8 + quad * 2 + (i & 1)][hq] = p[i];
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < kDecRows; ++r) {
      uint2 raw;
      asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(raw.x), "=r"(raw.y)
                   : "r"(vs + r * 256 + (((lane >> 1) ^ (r & 7)) << 4) + (lane & 1) * 8));
      const float2 v01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
      const float2 v23 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float pg = sm_p[warp][r][g];
        o[g][0] = fmaf(pg, v01.x, o[g][0]);
        o[g][1] = fmaf(pg, v01.y, o[g][1]);
        o[g][2] = fmaf(pg, v23.x, o[g][2]);
        o[g][3] = fmaf(pg, v23.y, o[g][3]);
      }
    }
  }
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  // ---- the four warps' sums, through the ring (every copy has landed: tiles that were asked for were waited for)
  cp_async_wait<0>();
  __syncthreads();
  float* sm_o = reinterpret_cast<float*>(dec_smem);        // [warp][G][128]
  __shared__ float sm_m[kDecWarps][8], sm_l[kDecWarps][8];
#pragma unroll
  for (int g = 0; g < G; ++g)
    *reinterpret_cast<float4*>(sm_o + (warp * G + g) * HD + lane * 4) = make_float4(o[g][0], o[g][1], o[g][2], o[g][3]);
  if (quad == 0) { sm_m[warp][hq] = m; sm_l[warp][hq] = l; }
  __syncthreads();
  const int col = threadIdx.x;
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const float mn = fmaxf(fmaxf(sm_m[0][g], sm_m[1][g]), fmaxf(sm_m[2][g], sm_m[3][g]));
    float acc = 0.f, ls = 0.f;
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) {
      const float c = mn == -INFINITY ? 0.f : exp2f(sm_m[w][g] - mn);
      acc += sm_o[(w * G + g) * HD + col] * c;
      ls += sm_l[w][g] * c;
    }
    if (out != nullptr) {                                  // the only stretch: nothing to merge
      out[b * o_sb + (long)(kvh * G + g) * o_sh + col] = __float2bfloat16_rn(ls > 0.f ? acc / ls : 0.f);
    } else {
      const long idx = (((long)b * H + kvh * G + g) * splits + split);
      part_o[idx * HD + col] = acc;
      if (col == 0) { part_ml[idx * 2] = mn; part_ml[idx * 2 + 1] = ls; }
    }
  }
}

// Merge of a head's stretches (at most 64): the sum of o relative to the row's maximum `mn`, and the row sum `ls`; thread = column.  The first
// sixteen stretches are asked for before their weights are known, and every warp gets all weights with one read per lane; walked one after the
// other, twice, they took 2 to 3 us more (8 x 8192 rows, 32 heads on 8, both kernels: 40.6 -> 38.9 us; 1 x 2048, 40 heads: 9.4 -> 8.7).
NXD_DEVICE float merge_stretches(const float* part_o, const float* part_ml, int bh, int splits, float& mn, float& ls) {
  const float2* ml = reinterpret_cast<const float2*>(part_ml) + (long)bh * splits;
  const float* po = part_o + (long)bh * splits * HD + threadIdx.x;
  const int lane = threadIdx.x & 31;
  float v[16];
#pragma unroll
  for (int s = 0; s < 16; ++s) v[s] = s < splits ? po[(long)s * HD] : 0.f;
  const float2 a0 = lane < splits ? ml[lane] : make_float2(-INFINITY, 0.f), a1 = lane + 32 < splits ? ml[lane + 32] : make_float2(-INFINITY, 0.f);
  mn = warp_max(fmaxf(a0.x, a1.x));
  const float c0 = mn == -INFINITY ? 0.f : exp2f(a0.x - mn), c1 = mn == -INFINITY ? 0.f : exp2f(a1.x - mn);
  ls = warp_sum(a0.y * c0 + a1.y * c1);
  float acc = 0.f;
#pragma unroll
  for (int s = 0; s < 16; ++s) acc += v[s] * __shfl_sync(0xffffffffu, c0, s);
#pragma unroll 8
  for (int s = 16; s < splits; ++s) acc += po[(long)s * HD] * __shfl_sync(0xffffffffu, s < 32 ? c0 : c1, s & 31);
  return acc;
}

__global__ void __launch_bounds__(HD) decode_combine_kernel(const float* part_o, const float* part_ml,
                                                            __nv_bfloat16* out, int splits, long o_sb, long o_sh,
                                                            int H) {
  pdl_trigger();
  pdl_wait();
  float mn, ls;
  const float acc = merge_stretches(part_o, part_ml, blockIdx.x, splits, mn, ls);
  const int b = blockIdx.x / H, h = blockIdx.x % H;
  out[b * o_sb + h * o_sh + threadIdx.x] = __float2bfloat16_rn(ls > 0.f ? acc / ls : 0.f);
}

// Same merge over the splits, but the result stays un-normalised: o (relative to the row maximum), the maximum (natural-log
// units) and the row sum — what a rank contributes to distributed flash-decoding, where the final normalisation happens after
// the cross-rank log-sum-exp merge (modules/attention/flash_decode.py).
__global__ void __launch_bounds__(HD) decode_combine_partial_kernel(const float* part_o, const float* part_ml,
                                                                    float* fin_o, float* fin_ml, int splits) {
  pdl_wait();
  float mn, ls;
  const float acc = merge_stretches(part_o, part_ml, blockIdx.x, splits, mn, ls);
  fin_o[(long)blockIdx.x * HD + threadIdx.x] = acc;
  if (threadIdx.x == 0) { fin_ml[blockIdx.x * 2] = mn * 0.6931471805599453f; fin_ml[blockIdx.x * 2 + 1] = ls; }
}

// While the kernel before it still runs (a norm, a rotation, the merge of an attention), the first bytes of its weights come to L2:
// 13B, one token, us: 324 with ordinary launches, 310.5 with dependent ones, 307.4 / 309.5 / 333 with 2 / 4 / 10 KB of a row ahead.
constexpr int kGemvAhead = 2048;

// y[m, n] = Σ_k x[m, k] · W[n, k]; one warp per output column n (8 columns per 256-thread CTA), M ≤ 8 rows of x kept hot in L1.
template <int M>
__global__ void __launch_bounds__(256) gemv_kernel(const __nv_bfloat16* x, const __nv_bfloat16* w, const __nv_bfloat16* residual, __nv_bfloat16* y,
                                                   int N, int K) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.x * 8 + warp;
  if (lane == 0 && n < N) prefetch_l2(w + (long)n * K, (uint32_t)min(K * 2, kGemvAhead));
  pdl_wait();
  if (n >= N) return;
  float acc[M];
#pragma unroll
  for (int m = 0; m < M; ++m) acc[m] = 0.f;
  const __nv_bfloat16* wr = w + (long)n * K;
#pragma unroll 4
  for (int k = lane * 8; k < K; k += 256) {
    const uint4 wv = *reinterpret_cast<const uint4*>(wr + k);       // weights stream through once
    const __nv_bfloat162* w2 = reinterpret_cast<const __nv_bfloat162*>(&wv);
    float wf[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(w2[i]); wf[2 * i] = f.x; wf[2 * i + 1] = f.y; }
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const uint4 xv = *reinterpret_cast<const uint4*>(x + (long)m * K + k);
      const __nv_bfloat162* x2 = reinterpret_cast<const __nv_bfloat162*>(&xv);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(x2[i]);
        acc[m] = fmaf(f.x, wf[2 * i], acc[m]);
        acc[m] = fmaf(f.y, wf[2 * i + 1], acc[m]);
      }
    }
  }
  pdl_trigger();       // not before: blocks that start beside this kernel's fill the SMs unevenly and stay there (8192 wide: 179 us -> 232 a token)
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const float v = warp_sum(acc[m]);
    if (lane == 0) {
      float r = v;
      if (residual) r += __bfloat162float(residual[(long)m * N + n]);
      y[(long)m * N + n] = __float2bfloat16_rn(r);
    }
  }
}

// Decode-time RoPE + KV-cache append in ONE launch (was ~25 tiny elementwise / index_put kernels per layer in the token-
// generation graph): q [B,H,D] rotated into q_out, k rotated and v copied into the cache row positions[b].  One warp per head
// row; cos/sin rows gathered by position.  HF rotate-half convention (csrc/elementwise.cu rope_kernel).
__global__ void __launch_bounds__(128) decode_rope_kv_kernel(const __nv_bfloat16* q, const __nv_bfloat16* k,
                                                            const __nv_bfloat16* v, const long* positions,
                                                            const float* cos_t, const float* sin_t,
                                                            __nv_bfloat16* q_out, __nv_bfloat16* kc,
                                                            __nv_bfloat16* vc, int B, int H, int Hkv, int D, int L,
                                                            long q_sb, long q_sh, long k_sb, long k_sh, long v_sb, long v_sh,
                                                            long c_sb, long c_ss, long c_sh) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int rows = B * (H + 2 * Hkv);
  pdl_trigger();
  pdl_wait();
  if (warp >= rows) return;
  const int b = warp / (H + 2 * Hkv), r = warp % (H + 2 * Hkv);
  long pos = positions[b];
  pos = pos < 0 ? 0 : (pos >= L ? L - 1 : pos);
  const int half = D / 2;
  if (r < H + Hkv) {                                   // q or k head: rotate
    const bool is_q = r < H;
    const int h = is_q ? r : r - H;
    const __nv_bfloat16* src = is_q ? q + b * q_sb + (long)h * q_sh : k + b * k_sb + (long)h * k_sh;
    __nv_bfloat16* dst = is_q ? q_out + ((long)b * H + h) * D : kc + b * c_sb + pos * c_ss + (long)h * c_sh;
    const float* cr = cos_t + pos * half;
    const float* sr = sin_t + pos * half;
    for (int c = lane; c < half; c += 32) {
      const float a = __bfloat162float(src[c]), bb = __bfloat162float(src[half + c]);
      const float cs = cr[c], sn = sr[c];
      dst[c] = __float2bfloat16_rn(a * cs - bb * sn);
      dst[half + c] = __float2bfloat16_rn(bb * cs + a * sn);
    }
  } else {                                             // v head: copy
    const int h = r - H - Hkv;
    const __nv_bfloat16* src = v + b * v_sb + (long)h * v_sh;
    __nv_bfloat16* dst = vc + b * c_sb + pos * c_ss + (long)h * c_sh;
    for (int c = lane; c < D; c += 32) dst[c] = src[c];
  }
}

}  // namespace

void decode_rope_kv(const void* q, const void* k, const void* v, const long* positions, const float* cos_t, const float* sin_t,
                    void* q_out, void* kc, void* vc, int B, int H, int Hkv, int D, int L, long q_sb, long q_sh, long k_sb, long k_sh,
                    long v_sb, long v_sh, long c_sb, long c_ss, long c_sh, cudaStream_t st) {
  const int rows = B * (H + 2 * Hkv);
  const int grid = (rows * 32 + 127) / 128;
  launch_dependent(decode_rope_kv_kernel, grid, 128, 0, st, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, positions,
                   cos_t, sin_t, (__nv_bfloat16*)q_out, (__nv_bfloat16*)kc, (__nv_bfloat16*)vc, B, H, Hkv, D, L,
                   q_sb, q_sh, k_sb, k_sh, v_sb, v_sh, c_sb, c_ss, c_sh);
}

// Stretches per (sequence, key/value head): about six blocks per SM in all, so that sequences of unequal length fill the GPU to
// the end (8 x 8192 rows, 8 key/value heads, with the merge: 41.0 us; three per SM 43.6, nine 42.3), and no stretch below 256 rows, where a block's
// start and the merge outweigh its reading (1 x 2048 rows, 40 heads, 128-row stretches a tenth slower, 64-row a third).  At most 64 (the merge).
int device_sm_count();
int decode_splits(int pairs, int L) {
  const int want = (6 * device_sm_count() + pairs - 1) / pairs;
  return std::max(1, std::min(std::min(want, 64), (L + 255) / 256));
}

void decode_attention(const void* q, const void* k, const void* v, const long* positions, void* out, float* part_o,
                      float* part_ml, int B, int H, int Hkv, int L, const long* ks, const long* vs, long q_sb, long q_sh,
                      long o_sb, long o_sh, float scale, int splits, cudaStream_t st, float* fin_o, float* fin_ml) {
  const int G = H / Hkv;
  dim3 grid(Hkv, B, splits);
  const float sl2 = scale * 1.4426950408889634f;
  const bool whole = splits == 1 && fin_o == nullptr;
  // Launches that three blocks per SM take at once are a few round trips to memory long, and need them deeper rather than more of them at a time.
  // Single heads' blocks copy the most and compute the least: in launches of 896 to 1280 of them, caches in memory, two stages took 0.89 to 1.02 of
  // the time of three (16 x 2048 rows, 8 heads: 20.7 us and 23.2; 16 x 4096, 40 heads: 144.6 and 148.2; 8 x 8192, 32 heads: 118.4 and 118.1;
  // 3 x 16384, 32 heads: 103.2 and 100.9), by no length of theirs in particular.
  const bool few = (long)Hkv * B * splits <= 3l * device_sm_count();
#define NXD_DEC_STAGES(Gv, Sv)                                                                                       \
  do {                                                                                                               \
    NXD_ALLOW_SMEM((decode_attn_kernel<Gv, Sv>), dec_smem_bytes(Sv));                                                  \
    launch_dependent(decode_attn_kernel<Gv, Sv>, grid, kDecThreads, dec_smem_bytes(Sv), st, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k, \
        (const __nv_bfloat16*)v, positions, part_o, part_ml, whole ? (__nv_bfloat16*)out : nullptr, B, H, Hkv, L,      \
        ks[0], ks[1], ks[2], vs[0], vs[1], vs[2], q_sb, q_sh, o_sb, o_sh, sl2, splits);                                \
  } while (0)
#define NXD_DEC(Gv) do { if (few) NXD_DEC_STAGES(Gv, 3); else NXD_DEC_STAGES(Gv, 2); } while (0)
  switch (G) {
    case 1: NXD_DEC(1); break;
    case 2: NXD_DEC(2); break;
    case 3: NXD_DEC(3); break;
    case 4: NXD_DEC(4); break;
    case 5: NXD_DEC(5); break;
    case 6: NXD_DEC(6); break;
    case 7: NXD_DEC(7); break;
    case 8: NXD_DEC(8); break;
    default: nxd_throw("decode_attention: unsupported GQA group size", __FILE__, __LINE__);
  }
#undef NXD_DEC
#undef NXD_DEC_STAGES
  if (fin_o != nullptr) launch_dependent(decode_combine_partial_kernel, B * H, HD, 0, st, part_o, part_ml, fin_o, fin_ml, splits);
  else if (!whole) launch_dependent(decode_combine_kernel, B * H, HD, 0, st, part_o, part_ml, (__nv_bfloat16*)out, splits, o_sb, o_sh, H);
  NXD_CUDA_CHECK(cudaGetLastError());
}

// Rows of x for which the vector kernel is the faster one (the figures stand in gemv_bf16)
static bool vector_rows(int M, int N, int K) {
  const bool tiny = (long)N * K <= ((long)M * K < 4096 ? 8l << 20 : (long)M * K < 8192 ? 4l << 20 : 0);
  return !((M >= 3 && !tiny) || (M == 2 && (long)N * K >= 28l << 20));
}

// y [M, I] = SwiGLU of x [M, K] · w [2 I, K]ᵀ for up to 8 rows; false: rows for the vector kernel, which is faster with a launch of SwiGLU behind it
// than with a gate and an up row a warp (a token of 13B: 310.9 us, and 313.2 on the same scale)
bool gemv_swiglu(const void* x, const void* w, void* y, int M, int I, int K, cudaStream_t st) {
  if (vector_rows(M, 2 * I, K)) return false;
  gemm_few_rows_swiglu(x, w, y, M, I, K, st);
  return true;
}

void gemv_bf16(const void* x, const void* w, const void* residual, void* y, int M, int N, int K, cudaStream_t st) {
  // From three rows on (two where the weights are large) the vector kernel is bound by its multiply-adds and loads of x, not by
  // the weights: 27648 x 5120, 1 / 2 / 4 / 8 rows: 41 / 50 / 86 / 162 us against 45 / 46 / 46 / 46 on the tensor cores; 5120 x 5120,
  // 2 rows: 12.2 against 13.2.  Small weights with short rows are done before a ring is filled: 1024 x 1024, 3 / 4 rows 8.2 against
  // 10.2, 512 x 512, 8 rows 8.2 against 10.2, 5632 x 1024, 3 rows 10.2 against 12.3; but 64 x 4096, 4 rows 17 against 11, 32000 x 512,
  // 4 rows 21 against 13, 5632 x 1024, 8 rows 18 against 11.
  if (!vector_rows(M, N, K) && N % 8 == 0 && K % 8 == 0 &&
      (((uintptr_t)x | (uintptr_t)w | (uintptr_t)y | (uintptr_t)residual) % 16) == 0)
    return gemm_few_rows(x, w, residual, y, M, N, K, 0, st);
  const int grid = (N + 7) / 8;
#define NXD_GEMV(Mv)                                                                                                \
  launch_dependent(gemv_kernel<Mv>, grid, 256, 0, st, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (const __nv_bfloat16*)residual, \
                   (__nv_bfloat16*)y, N, K)
  switch (M) {
    case 1: NXD_GEMV(1); break;
    case 2: NXD_GEMV(2); break;
    case 3: NXD_GEMV(3); break;
    case 4: NXD_GEMV(4); break;
    case 5: NXD_GEMV(5); break;
    case 6: NXD_GEMV(6); break;
    case 7: NXD_GEMV(7); break;
    case 8: NXD_GEMV(8); break;
    default: nxd_throw("gemv_bf16: M must be 1..8", __FILE__, __LINE__);
  }
#undef NXD_GEMV
  NXD_CUDA_CHECK(cudaGetLastError());
}

}  // namespace nxd

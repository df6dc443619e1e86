// Rows of routed experts in expert order: where each (token, choice) goes, the copy there, and the weighted sum back.
//   moe_slots          expert ids [T, k] → slot of each choice, token of each slot, expert of each row block, block prefix sums
//   moe_gather         x [T, H] → rows in slot order (padding rows zero)
//   moe_combine        out[t] = sum_j w[t, e_j] · y[slot(t, j)]      (w optional)
//   moe_combine_grad   dy[slot] = w[t, e] · g[t],  dw[t, e] += <g[t], y[slot]>
//   moe_normalize      w[t] = the chosen affinities of t divided by their sum, and the way back
// All are bound by memory: every row is read once and written once in 16-byte packets, sums are fp32 in a fixed order, and
// nothing but the affinity gradient (a dot product per slot) uses atomics.  4096 tokens, two of eight experts, hidden 4096:
// gather 17 us, combine 20, its gradient 31; the index / mul / index_add passes and their sorted scatter backward that they
// replace took 6.1 of the layer's 8.6 ms.
#include "common.cuh"
#include "kernels.h"

namespace nxd {
namespace {

constexpr int kSlotThreads = 1024;
constexpr int kMaxExperts = 256;

// Every block counts the whole list (and, apart, what lies before its own chunk), so the chunks need no exchange; then it
// places its chunk in stable order.  8192 choices: 8 us; one block alone took 18, and 83 for 40 thousand: a serial chain of
// block-wide steps of 1024 choices.
template <typename IdxT, typename OutT>
__global__ void __launch_bounds__(kSlotThreads) moe_slots_kernel(const IdxT* __restrict__ expert_index, long n, int k, int E, int B,
                                                                 int nb, long chunk, OutT* __restrict__ block_to_expert,
                                                                 OutT* __restrict__ slot_token, OutT* __restrict__ counts_out,
                                                                 int* __restrict__ seg, int* __restrict__ slot_of) {
  __shared__ int total[kMaxExperts], next[kMaxExperts], first[kMaxExperts + 1];
  __shared__ int wc[32][kMaxExperts];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long c0 = (long)blockIdx.x * chunk, c1 = min(n, c0 + chunk);
  for (int e = tid; e < E; e += kSlotThreads) total[e] = next[e] = 0;
  __syncthreads();
  for (long i0 = 0; i0 < n; i0 += kSlotThreads) {
    const long i = i0 + tid;
    int e = i < n ? (int)expert_index[i] : -1;
    if (e < 0 || e >= E) e = -1;
    const unsigned same = __match_any_sync(0xffffffffu, e);
    const unsigned before = __ballot_sync(0xffffffffu, i < c0) & same;
    if (e >= 0 && (same & ((1u << lane) - 1u)) == 0) {
      atomicAdd(&total[e], __popc(same));
      if (before) atomicAdd(&next[e], __popc(before));
    }
  }
  __syncthreads();
  if (warp == 0) {                                          // first row block of every expert
    int sum = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane;
      const int own = e < E ? (total[e] + B - 1) / B : 0;
      int v = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
      }
      if (e < E) first[e] = sum + v - own;
      sum += __shfl_sync(0xffffffffu, v, 31);
    }
    if (lane == 0) first[E] = sum;
  }
  __syncthreads();
  for (int e = tid; e < E; e += kSlotThreads) next[e] += first[e] * B;
  if (blockIdx.x == 0) {
    for (int e = tid; e < E; e += kSlotThreads) {
      if (counts_out) counts_out[e] = total[e];
      for (int b = first[e]; b < first[e + 1] && b < nb; ++b) block_to_expert[b] = e;
    }
    for (int b = first[E] + tid; b < nb; b += kSlotThreads) block_to_expert[b] = E - 1;      // no tokens behind here
    if (seg) for (int e = tid; e <= E; e += kSlotThreads) seg[e] = first[e];
  }
  // padding slots of the experts (one warp each) and of the blocks behind them, shared by all blocks
  const int gwarp = blockIdx.x * 32 + warp, warps = gridDim.x * 32;
  for (int e = gwarp; e <= E; e += warps) {
    const long lo = e < E ? (long)first[e] * B + total[e] : (long)first[E] * B;
    const long hi = min((long)nb * B, e < E ? (long)first[e + 1] * B : (long)nb * B);
    for (long s = lo + lane; s < hi; s += 32) slot_token[s] = -1;
  }
  __syncthreads();
  for (long at = c0; at < c1; at += kSlotThreads) {
    for (int j = tid; j < 32 * E; j += kSlotThreads) wc[j / E][j % E] = 0;
    __syncthreads();
    const long i = at + tid;
    int e = i < c1 ? (int)expert_index[i] : -1;
    if (e < 0 || e >= E) e = -1;
    const unsigned same = __match_any_sync(0xffffffffu, e);
    const int rank = __popc(same & ((1u << lane) - 1u));
    if (e >= 0 && rank == 0) wc[warp][e] = __popc(same);
    __syncthreads();
    for (int x = tid; x < E; x += kSlotThreads) {           // counts of the 32 warps → their first slots
      int run = next[x];
#pragma unroll
      for (int w = 0; w < 32; ++w) { const int c = wc[w][x]; wc[w][x] = run; run += c; }
      next[x] = run;
    }
    __syncthreads();
    if (i < c1) {
      const long slot = e >= 0 ? (long)wc[warp][e] + rank : -1;
      const bool ok = slot >= 0 && slot < (long)nb * B;
      if (ok) slot_token[slot] = (OutT)(i / k);
      if (slot_of) slot_of[i] = ok ? (int)slot : -1;
    }
    __syncthreads();
  }
}

constexpr int kRowThreads = 128;

__global__ void __launch_bounds__(kRowThreads) moe_gather_kernel(const __nv_bfloat16* __restrict__ x, const int* __restrict__ slot_token,
                                                                 const int* __restrict__ used_blocks, __nv_bfloat16* __restrict__ out,
                                                                 int H, int B) {
  const long slot = blockIdx.x;
  if (slot >= (long)*used_blocks * B) return;
  const int t = slot_token[slot], nvec = H / 8;
  const uint4* src = reinterpret_cast<const uint4*>(x + (long)max(t, 0) * H);
  uint4* dst = reinterpret_cast<uint4*>(out + slot * H);
#pragma unroll 4
  for (int v = threadIdx.x; v < nvec; v += kRowThreads) dst[v] = t >= 0 ? __ldg(src + v) : make_uint4(0, 0, 0, 0);
}

template <bool WEIGHTED>
__global__ void __launch_bounds__(kRowThreads) moe_combine_kernel(const __nv_bfloat16* __restrict__ y, const int* __restrict__ slot_of,
                                                                  const long* __restrict__ expert_index, const float* __restrict__ w,
                                                                  __nv_bfloat16* __restrict__ out, int H, int E, int k) {
  const long t = blockIdx.x;
  const int nvec = H / 8;
  for (int v = threadIdx.x; v < nvec; v += kRowThreads) {
    float acc[8] = {};
#pragma unroll 4
    for (int j = 0; j < k; ++j) {
      const int slot = slot_of[t * k + j];
      if (slot < 0) continue;
      const float a = WEIGHTED ? w[t * E + expert_index[t * k + j]] : 1.f;
      Pack16<__nv_bfloat16> p;
      p.load_nc(y + (long)slot * H + v * 8);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = fmaf(a, p.f(i), acc[i]);
    }
    Pack16<__nv_bfloat16> o;
#pragma unroll
    for (int i = 0; i < 8; ++i) o.set(i, acc[i]);
    o.store(out + t * H + v * 8);
  }
}

__global__ void __launch_bounds__(kRowThreads) moe_combine_grad_kernel(const __nv_bfloat16* __restrict__ g, const __nv_bfloat16* __restrict__ y,
                                                                       const int* __restrict__ slot_token, const int* __restrict__ block_expert,
                                                                       const int* __restrict__ used_blocks, const float* __restrict__ w,
                                                                       __nv_bfloat16* __restrict__ dy, float* __restrict__ dw, int H, int E,
                                                                       int B) {
  __shared__ float red[32];
  const long slot = blockIdx.x;
  if (slot >= (long)*used_blocks * B) return;
  const int t = slot_token[slot], e = block_expert[slot / B], nvec = H / 8;
  const float a = t >= 0 ? w[(long)t * E + e] : 0.f;
  float dot = 0.f;
#pragma unroll 4
  for (int v = threadIdx.x; v < nvec; v += kRowThreads) {
    Pack16<__nv_bfloat16> o, p, q;
    *reinterpret_cast<uint4*>(o.v) = make_uint4(0, 0, 0, 0);
    if (t >= 0) {
      p.load_nc(g + (long)t * H + v * 8);
      q.load_nc(y + slot * H + v * 8);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        dot = fmaf(p.f(i), q.f(i), dot);
        o.set(i, a * p.f(i));
      }
    }
    o.store(dy + slot * H + v * 8);
  }
  if (t < 0) return;
  dot = block_sum(dot, red);
  if (threadIdx.x == 0) atomicAdd(dw + (long)t * E + e, dot);
}

// Affinities times the mask of the chosen experts, divided by their sum (at least kLeastSum); GRAD: the gradient of the affinities out of that of
// the quotients.  One warp per token.  Both ways a dozen launches on small tensors otherwise (fill, scatter, multiply, sum, clamp, divide and
// back), 50 us of a layer of 4096 tokens; two launches of 3 us so.
constexpr float kLeastSum = 1e-9f;
template <bool GRAD>
__global__ void __launch_bounds__(kRowThreads) moe_normalize_kernel(const float* __restrict__ aff, const long* __restrict__ expert_index,
                                                                    const float* __restrict__ gw, float* __restrict__ out, int T, int E, int k) {
  const int t = blockIdx.x * (kRowThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= T) return;
  const float *a = aff + (long)t * E, *g = gw + (long)t * E;
  const long* idx = expert_index + (long)t * k;
  constexpr int kPer = kMaxExperts / 32;                   // experts of a lane
  float v[kPer], m[kPer], sum = 0.f, dot = 0.f;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = i * 32 + lane;
    v[i] = m[i] = 0.f;
    if (i * 32 >= E) continue;
    for (int j = 0; j < k; ++j) m[i] = idx[j] == e ? 1.f : m[i];
    if (e < E) v[i] = a[e] * m[i];                         // a product: NaN where an affinity is, chosen or not
    sum += v[i];
    if (GRAD && e < E) dot = fmaf(g[e], v[i], dot);
  }
  sum = warp_sum(sum);
  const bool small = sum < kLeastSum;                      // then the sum counts as kLeastSum and has no gradient
  const float s = small ? kLeastSum : sum;
  float dsum = 0.f;
  if constexpr (GRAD) dsum = small ? 0.f : -__fdiv_rn(__fdiv_rn(warp_sum(dot), s), s);
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = i * 32 + lane;
    if (e < E) out[(long)t * E + e] = GRAD ? (__fdiv_rn(g[e], s) + dsum) * m[i] : __fdiv_rn(v[i], s);
  }
}

}  // namespace

void moe_normalize(const float* aff, const long* expert_index, const float* gw, float* out, int T, int E, int k, cudaStream_t st) {
  if ((long)T * E == 0) return;
  if (E > kMaxExperts) nxd_throw("moe_normalize: at most 256 experts", __FILE__, __LINE__);
  const int grid = (T + kRowThreads / 32 - 1) / (kRowThreads / 32);
  if (gw) moe_normalize_kernel<true><<<grid, kRowThreads, 0, st>>>(aff, expert_index, gw, out, T, E, k);
  else moe_normalize_kernel<false><<<grid, kRowThreads, 0, st>>>(aff, expert_index, gw, out, T, E, k);
  NXD_CUDA_CHECK(cudaGetLastError());
}

// Chunks of the list per block: at most 32 blocks, since every block counts the whole list.
template <typename OutT>
static void slots(const void* idx, bool idx64, long n, int k, int E, int B, int nb, OutT* b2e, OutT* slot_token, OutT* counts, int* seg,
                  int* slot_of, cudaStream_t st) {
  if (E > kMaxExperts) nxd_throw("moe_block_metadata: at most 256 experts", __FILE__, __LINE__);
  const long chunks = (n + kSlotThreads - 1) / kSlotThreads;
  const int grid = (int)(chunks < 1 ? 1 : chunks < 32 ? chunks : 32);
  const long chunk = (chunks + grid - 1) / grid * kSlotThreads;
  if (idx64) moe_slots_kernel<long, OutT><<<grid, kSlotThreads, 0, st>>>((const long*)idx, n, k, E, B, nb, chunk, b2e, slot_token, counts, seg, slot_of);
  else moe_slots_kernel<int, OutT><<<grid, kSlotThreads, 0, st>>>((const int*)idx, n, k, E, B, nb, chunk, b2e, slot_token, counts, seg, slot_of);
  NXD_CUDA_CHECK(cudaGetLastError());
}

void moe_block_metadata(const void* expert_index, bool idx64, long n, int k, int E, int B, int nb, long* block_to_expert, long* tp2id,
                        long* counts, cudaStream_t st) {
  slots<long>(expert_index, idx64, n, k, E, B, nb, block_to_expert, tp2id, counts, nullptr, nullptr, st);
}

void moe_slots(const long* expert_index, long n, int k, int E, int B, int nb, int* block_expert, int* slot_token, int* seg, int* slot_of,
               cudaStream_t st) {
  slots<int>(expert_index, true, n, k, E, B, nb, block_expert, slot_token, (int*)nullptr, seg, slot_of, st);
}

void moe_gather(const void* x, const int* slot_token, const int* used_blocks, void* out, int H, int B, int rows, cudaStream_t st) {
  if (rows == 0) return;
  moe_gather_kernel<<<rows, kRowThreads, 0, st>>>((const __nv_bfloat16*)x, slot_token, used_blocks, (__nv_bfloat16*)out, H, B);
  NXD_CUDA_CHECK(cudaGetLastError());
}

void moe_combine(const void* y, const int* slot_of, const long* expert_index, const float* w, void* out, int T, int H, int E, int k,
                 cudaStream_t st) {
  if (T == 0) return;
  if (w) moe_combine_kernel<true><<<T, kRowThreads, 0, st>>>((const __nv_bfloat16*)y, slot_of, expert_index, w, (__nv_bfloat16*)out, H, E, k);
  else moe_combine_kernel<false><<<T, kRowThreads, 0, st>>>((const __nv_bfloat16*)y, slot_of, expert_index, w, (__nv_bfloat16*)out, H, E, k);
  NXD_CUDA_CHECK(cudaGetLastError());
}

void moe_combine_grad(const void* g, const void* y, const int* slot_token, const int* block_expert, const int* used_blocks, const float* w,
                      void* dy, float* dw, int H, int E, int B, int rows, cudaStream_t st) {
  if (rows == 0) return;
  moe_combine_grad_kernel<<<rows, kRowThreads, 0, st>>>((const __nv_bfloat16*)g, (const __nv_bfloat16*)y, slot_token, block_expert,
                                                        used_blocks, w, (__nv_bfloat16*)dy, dw, H, E, B);
  NXD_CUDA_CHECK(cudaGetLastError());
}

}  // namespace nxd

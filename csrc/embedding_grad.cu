// Gradient of an embedding table:
//   out[id] += sum of gy[t] over all t with ids[t] == id       (fp32, in a fixed order: the same sum on every run)
//
// Tokens repeat: padding, frequent words, and on a vocabulary shard every token of another rank, which looks up row 0.  So the tokens
// are put in the order of their ids first, and the rows of one id are summed in stretches of 64, each by blocks of its own; an id
// of one stretch goes straight to `out`, the sums of longer ones to a workspace that a last kernel adds up.  Bound by reading gy and
// by the latency of a few dependent loads.  32000 x 4096 table, 2048 tokens: 30 us and 39 to zero the table; 32768 tokens 394 and 39.  One
// block per id, row after row, took 2.6 ms for 4096 equal tokens and 20 ms for 32768, with the gradient buffer's update; now 0.25 and 0.78.
#include "common.cuh"
#include "kernels.h"

namespace nxd {
namespace {

constexpr int kStretch = 64;
constexpr int kThreads = 256;                   // one packet of 8 columns each
constexpr int kTokens = 32, kSlices = 32;       // of a sorting block: its tokens, and the warps that share the list they are compared with
constexpr int kTile = kTokens * kSlices;

// order[p]: the token at place p, ids ascending and equal ids by token; first[p]: the place of the first token of its id.  A token's
// place is the number of smaller ids and of equal ones before it: T * T comparisons, a few for each thread (32768 tokens are the limit
// of its caller), no serial chain of passes.  Ids outside 0 .. V-1 come first, as -1.
__global__ void __launch_bounds__(kTile) embedding_order_kernel(const long* __restrict__ ids, int* __restrict__ order, int* __restrict__ first,
                                                                int T, long V) {
  __shared__ __align__(16) int keys[kTile];
  __shared__ int2 count[kSlices][kTokens];
  const int tid = threadIdx.x, slice = tid / kTokens, at = tid % kTokens, t = blockIdx.x * kTokens + at;
  auto key = [&](int u) { const long id = ids[u]; return id < 0 || id >= V ? -1 : (int)id; };
  const int mine = t < T ? key(t) : -1;
  int less = 0, equal = 0;                      // equal ids: of tokens before this one
  for (int u0 = 0; u0 < T; u0 += kTile) {
    keys[tid] = u0 + tid < T ? key(u0 + tid) : 0x7fffffff;        // beyond the list: neither smaller nor equal
    __syncthreads();
    const int lo = slice * kTokens;
    const int4* k4 = reinterpret_cast<const int4*>(keys + lo);
    if (u0 + lo < (int)blockIdx.x * kTokens) {
#pragma unroll 8
      for (int i = 0; i < kTokens / 4; ++i) {
        const int4 k = k4[i];
        less += (k.x < mine) + (k.y < mine) + (k.z < mine) + (k.w < mine);
        equal += (k.x == mine) + (k.y == mine) + (k.z == mine) + (k.w == mine);
      }
    } else {                                    // the block's own tokens, or tokens behind them
      const bool own = u0 + lo == (int)blockIdx.x * kTokens;
#pragma unroll 8
      for (int i = 0; i < kTokens / 4; ++i) {
        const int4 k = k4[i];
        less += (k.x < mine) + (k.y < mine) + (k.z < mine) + (k.w < mine);
        if (own) equal += (k.x == mine && 4 * i < at) + (k.y == mine && 4 * i + 1 < at) + (k.z == mine && 4 * i + 2 < at) + (k.w == mine && 4 * i + 3 < at);
      }
    }
    __syncthreads();
  }
  count[slice][at] = make_int2(less, equal);
  __syncthreads();
  if (slice == 0 && t < T) {
#pragma unroll 8
    for (int s = 1; s < kSlices; ++s) { less += count[s][at].x; equal += count[s][at].y; }
    order[less + equal] = t;
    first[less + equal] = less;
  }
}

template <typename Out>
NXD_DEVICE void add_to_row(Out* __restrict__ row, const float (&acc)[8]) {
#pragma unroll
  for (int c = 0; c < 8; c += Pack16<Out>::N) {
    Pack16<Out> o;
    o.load(row + c);
#pragma unroll
    for (int j = 0; j < Pack16<Out>::N; ++j) o.set(j, o.f(j) + acc[c + j]);
    o.store(row + c);
  }
}

// One block per place and 2048 columns; places that start no stretch leave.  Row of `part` for the stretch that starts at p: two per
// kStretch places, since there a single id of several stretches begins and a single one goes on.
template <typename Out>
__global__ void __launch_bounds__(kThreads) embedding_sum_kernel(const long* __restrict__ ids, const int* __restrict__ order,
                                                                 const int* __restrict__ first, const __nv_bfloat16* __restrict__ gy,
                                                                 Out* __restrict__ out, float* __restrict__ part, int T, int H, long V) {
  __shared__ int rows[kStretch];
  const int p = blockIdx.x, f = first[p], tid = threadIdx.x;
  if ((p - f) % kStretch) return;
  const long id = ids[order[p]];
  if (id < 0 || id >= V) return;
  const bool in = tid < kStretch && p + tid < T && first[p + tid] == f;
  if (in) rows[tid] = order[p + tid];
  const int n = __syncthreads_count(in);
  const bool several = p > f || (p + kStretch < T && first[p + kStretch] == f);
  const int c = (blockIdx.y * kThreads + tid) * 8;
  if (c >= H) return;
  float acc[8] = {};
  auto add = [&](const Pack16<__nv_bfloat16>& x) {
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] += x.f(j);
  };
  int k = 0;
  constexpr int U = 8;                          // rows in flight
  for (; k + U <= n; k += U) {
    Pack16<__nv_bfloat16> x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) x[u].load_nc(gy + (size_t)rows[k + u] * H + c);
#pragma unroll
    for (int u = 0; u < U; ++u) add(x[u]);
  }
  for (; k < n; ++k) { Pack16<__nv_bfloat16> x; x.load_nc(gy + (size_t)rows[k] * H + c); add(x); }
  if (!several) return add_to_row(out + (size_t)id * H + c, acc);
  float4* o = reinterpret_cast<float4*>(part + (size_t)(p / kStretch * 2 + (p == f)) * H + c);
  o[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
  o[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
}

// One block per kStretch places and 2048 columns: the id of several stretches that begins there, if any.
template <typename Out>
__global__ void __launch_bounds__(kThreads) embedding_merge_kernel(const long* __restrict__ ids, const int* __restrict__ order,
                                                                   const int* __restrict__ first, const float* __restrict__ part,
                                                                   Out* __restrict__ out, int T, int H, long V) {
  __shared__ int begin;
  const int tid = threadIdx.x, q = blockIdx.x * kStretch + tid;
  if (tid == 0) begin = -1;
  __syncthreads();
  if (tid < kStretch && q + kStretch < T && first[q] == q && first[q + kStretch] == q) begin = q;
  __syncthreads();
  const int p = begin, c = (blockIdx.y * kThreads + tid) * 8;
  if (p < 0 || c >= H) return;
  const long id = ids[order[p]];
  if (id < 0 || id >= V) return;
  float acc[8] = {};
#pragma unroll 4
  for (int s = p; s < T && first[s] == p; s += kStretch) {
    const float4* o = reinterpret_cast<const float4*>(part + (size_t)(s / kStretch * 2 + (s == p)) * H + c);
    const float4 a = o[0], b = o[1];
    acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
    acc[4] += b.x; acc[5] += b.y; acc[6] += b.z; acc[7] += b.w;
  }
  add_to_row(out + (size_t)id * H + c, acc);
}

template <typename Out>
void launch(const long* ids, const void* gy, Out* out, int* order, int* first, float* part, int T, int H, long V, cudaStream_t st) {
  const int cols = (H + 8 * kThreads - 1) / (8 * kThreads);
  embedding_order_kernel<<<(T + kTokens - 1) / kTokens, kTile, 0, st>>>(ids, order, first, T, V);
  embedding_sum_kernel<<<dim3(T, cols), kThreads, 0, st>>>(ids, order, first, (const __nv_bfloat16*)gy, out, part, T, H, V);
  if (T > kStretch) embedding_merge_kernel<<<dim3((T + kStretch - 1) / kStretch, cols), kThreads, 0, st>>>(ids, order, first, part, out, T, H, V);
}

}  // namespace

// floats of workspace: places and firsts of the tokens, padded to 16 bytes, and the stretches' sums
size_t embedding_grad_workspace(int T, int H) { return (size_t)(T + 3) / 4 * 8 + (T > kStretch ? (size_t)(T + kStretch - 1) / kStretch * 2 * H : 0); }

void embedding_grad(const long* ids, const void* gy, void* out, int out_dt, float* workspace, int T, int H, long V, cudaStream_t st) {
  if (T == 0) return;
  if (V > 0x7fffffff) nxd_throw("embedding_grad: at most 2^31 - 1 rows", __FILE__, __LINE__);
  int *order = reinterpret_cast<int*>(workspace), *first = order + (T + 3) / 4 * 4;
  float* part = workspace + (size_t)(T + 3) / 4 * 8;
  if (out_dt == kBF16) launch(ids, gy, (__nv_bfloat16*)out, order, first, part, T, H, V, st);
  else launch(ids, gy, (float*)out, order, first, part, T, H, V, st);
  NXD_CUDA_CHECK(cudaGetLastError());
}

}  // namespace nxd

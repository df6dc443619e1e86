// Row-wise selection kernels for on-device sampling (roles of the reference's NKI `cascaded_max` K10, `nkilib.core.topk`
// K11 and the torch_neuronx TopK / Argmax custom calls K12 — operators/argmax.py:129, operators/topk.py:17-21,
// utils/sampling.py:50-60).  A vocab(-shard) row is a one-pass HBM-bound reduction: one CTA per row, 16-byte loads,
// ties resolved to the smallest index (torch.argmax / torch.topk order on equal values is unspecified; the distributed
// wrappers in operators/ rely on "smallest global index wins").
//   row_argmax   x [R, V] → value fp32 [R], index int64 [R] (+ index_offset: global id of this rank's first column)
//   row_topk     x [R, V] → values fp32 [R, k], indices int64 [R, k], sorted descending; k <= 128, V*4 bytes <= 200 KB:
//                the row is staged once in shared memory as fp32 and k block-wide arg-max passes pick the winners.
#include <cfloat>

#include "common.cuh"
#include "kernels.h"

namespace nxd {

namespace {

struct ValIdx { float v; int i; };

NXD_DEVICE ValIdx better(ValIdx a, ValIdx b) {           // larger value, then smaller index
  return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a;
}
NXD_DEVICE ValIdx warp_best(ValIdx x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ValIdx y;
    y.v = __shfl_xor_sync(0xffffffffu, x.v, o);
    y.i = __shfl_xor_sync(0xffffffffu, x.i, o);
    x = better(x, y);
  }
  return x;
}
NXD_DEVICE ValIdx block_best(ValIdx x, ValIdx* smem) {    // smem: >= 32 entries; result valid in all threads
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  x = warp_best(x);
  __syncthreads();
  if (lane == 0) smem[warp] = x;
  __syncthreads();
  ValIdx r = lane < nw ? smem[lane] : ValIdx{-FLT_MAX, 0x7fffffff};
  r = warp_best(r);
  return r;
}

template <typename T>
__global__ void __launch_bounds__(256) row_argmax_kernel(const T* __restrict__ x, float* __restrict__ val, long* __restrict__ idx,
                                                         int V, long row_stride, long index_offset) {
  __shared__ ValIdx red[32];
  const T* row = x + (long)blockIdx.x * row_stride;
  ValIdx best{-FLT_MAX, 0x7fffffff};
  constexpr int N = 16 / sizeof(T);
  const bool vec_ok = ((uintptr_t)row % 16 == 0);
  const int nvec = vec_ok ? V / N : 0;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    Pack16<T> p;
    p.load(row + (long)v * N);
#pragma unroll
    for (int j = 0; j < N; ++j) best = better(best, ValIdx{p.f(j), v * N + j});
  }
  for (int c = nvec * N + threadIdx.x; c < V; c += blockDim.x) best = better(best, ValIdx{to_f32<T>(row[c]), c});
  best = block_best(best, red);
  if (threadIdx.x == 0) { val[blockIdx.x] = best.v; idx[blockIdx.x] = (long)best.i + index_offset; }
}

template <typename T>
__global__ void __launch_bounds__(256) row_topk_kernel(const T* __restrict__ x, float* __restrict__ vals, long* __restrict__ idxs,
                                                       int V, int k, long row_stride, long index_offset) {
  extern __shared__ float srow[];
  __shared__ ValIdx red[32];
  const T* row = x + (long)blockIdx.x * row_stride;
  for (int c = threadIdx.x; c < V; c += blockDim.x) srow[c] = to_f32<T>(row[c]);
  __syncthreads();
  for (int j = 0; j < k; ++j) {
    ValIdx best{-FLT_MAX, 0x7fffffff};
    for (int c = threadIdx.x; c < V; c += blockDim.x) best = better(best, ValIdx{srow[c], c});
    best = block_best(best, red);
    if (threadIdx.x == 0) {
      vals[(long)blockIdx.x * k + j] = best.v;
      idxs[(long)blockIdx.x * k + j] = (long)best.i + index_offset;
      if (best.i < V) srow[best.i] = -FLT_MAX;
    }
    __syncthreads();
  }
}

}  // namespace

void row_argmax(const void* x, float* val, long* idx, int rows, int V, long row_stride, long index_offset, int dt, cudaStream_t st) {
  if (rows == 0) return;
  if (dt == kBF16) row_argmax_kernel<__nv_bfloat16><<<rows, 256, 0, st>>>((const __nv_bfloat16*)x, val, idx, V, row_stride, index_offset);
  else if (dt == kF16) row_argmax_kernel<__half><<<rows, 256, 0, st>>>((const __half*)x, val, idx, V, row_stride, index_offset);
  else row_argmax_kernel<float><<<rows, 256, 0, st>>>((const float*)x, val, idx, V, row_stride, index_offset);
  NXD_CUDA_CHECK(cudaGetLastError());
}

bool row_topk_supported(int V, int k) { return k >= 1 && k <= 128 && (size_t)V * 4 <= 200 * 1024 && k <= V; }

void row_topk(const void* x, float* vals, long* idxs, int rows, int V, int k, long row_stride, long index_offset, int dt,
              cudaStream_t st) {
  if (rows == 0) return;
  if (!row_topk_supported(V, k)) nxd_throw("row_topk: k <= 128 and a row of at most 51200 elements", __FILE__, __LINE__);
  const size_t smem = (size_t)V * 4;
#define NXD_TOPK(T)                                                                                              \
  do {                                                                                                           \
    auto kern = row_topk_kernel<T>;                                                                              \
    if (smem > 48 * 1024) NXD_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
    kern<<<rows, 256, smem, st>>>((const T*)x, vals, idxs, V, k, row_stride, index_offset);                      \
  } while (0)
  if (dt == kBF16) NXD_TOPK(__nv_bfloat16);
  else if (dt == kF16) NXD_TOPK(__half);
  else NXD_TOPK(float);
#undef NXD_TOPK
  NXD_CUDA_CHECK(cudaGetLastError());
}

}  // namespace nxd

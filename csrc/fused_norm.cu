// Residual-add fused with RMSNorm (sm_100a, HBM-bound: one pass, 16-byte accesses, fp32 math).
//
//   forward :  h = x + r                      (the updated residual stream, written once)
//              y = h * rsqrt(mean(h^2) + eps) * w
//   backward:  dh = gh + rstd * (gy*w - hhat * mean_H(gy*w*hhat))     (gh: gradient arriving on the residual path)
//              dw = sum_rows gy * hhat                                   dx = dr = dh
//
// Unfused this is an add kernel (read x, r; write h) plus the norm (read h; write y) = 5 row passes forward and, backward,
// the norm backward (read gy, h; write d) plus an add (read d, gh; write dh) = 6; fused: 4 and 4.
// The forward math is that of rmsnorm_fwd_kernel (elementwise.cu), the backward kernel serves both norms; h is rounded to the storage dtype
// BEFORE the statistics so that y is exactly rmsnorm(h_stored), i.e. bit-compatible with the unfused sequence.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace nxd {

// WIDE: rows of more than 256 * MAXV packets; a kernel of its own, since its second loops cost the others registers (bf16: 66 instead
// of 48; 8192 x 5120: 74 us instead of 57).
template <typename T, int MAXV, bool WIDE>
__global__ void __launch_bounds__(256) add_rmsnorm_fwd_kernel(const T* __restrict__ x, const T* __restrict__ r,
                                                              const T* __restrict__ w, T* __restrict__ h,
                                                              T* __restrict__ y, float* __restrict__ rstd_out, int H,
                                                              float eps) {
  using P = Pack16<T>;
  constexpr int N = P::N;
  __shared__ float red[32];
  const int row = blockIdx.x;
  const size_t base = (size_t)row * H;
  const int nvec = H / N;
  P cache[MAXV];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      P px, pr;
      px.load(x + base + v * N);
      pr.load(r + base + v * N);
#pragma unroll
      for (int j = 0; j < N; ++j) {
        cache[i].set(j, px.f(j) + pr.f(j));
        const float f = cache[i].f(j);          // the rounded value: statistics of what is stored
        ss += f * f;
      }
      cache[i].store(h + base + v * N);
    }
  }
  // beyond what the registers hold: the second pass reads the stored sum again
  for (int v = threadIdx.x + MAXV * blockDim.x; WIDE && v < nvec; v += blockDim.x) {
    P px, pr;
    px.load(x + base + v * N);
    pr.load(r + base + v * N);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      px.set(j, px.f(j) + pr.f(j));
      const float f = px.f(j);
      ss += f * f;
    }
    px.store(h + base + v * N);
  }
  ss = block_sum(ss, red);
  const float rstd = rsqrtf(ss / (float)H + eps);
  if (threadIdx.x == 0) rstd_out[row] = rstd;
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      P pw, po;
      pw.load_nc(w + v * N);
#pragma unroll
      for (int j = 0; j < N; ++j) po.set(j, cache[i].f(j) * rstd * pw.f(j));
      po.store(y + base + v * N);
    }
  }
  for (int v = threadIdx.x + MAXV * blockDim.x; WIDE && v < nvec; v += blockDim.x) {
    P p, pw, po;
    p.load(h + base + v * N);
    pw.load_nc(w + v * N);
#pragma unroll
    for (int j = 0; j < N; ++j) po.set(j, p.f(j) * rstd * pw.f(j));
    po.store(y + base + v * N);
  }
}

// Backward of both norms (RES: with the gradient arriving on the residual path).  Persistent blocks stride over rows; each thread
// owns fixed columns, so its part of dW lives in registers across rows.  Bound by HBM if enough bytes are in flight: the rows of
// the next step (up to three 16-byte packets per thread) are loaded before this step's sum is reduced, and the sum costs one
// barrier (two alternating sets of partials).  8192 x 4096, bf16, with the residual path: 58 us (41 for its bytes), 95 with loads
// behind two barriers per row; the sum of the parts 3.5 us.
template <typename T, int VPT, bool RES>
__global__ void __launch_bounds__(512, VPT == 1 ? 2 : 1) norm_bwd_kernel(const T* __restrict__ gy, const T* __restrict__ gh,
                                                                         const T* __restrict__ h, const T* __restrict__ w,
                                                                         const float* __restrict__ rstd, T* __restrict__ dh,
                                                                         float* __restrict__ partial_dw, int rows, int H) {
  using P = Pack16<T>;
  constexpr int N = P::N;
  __shared__ float red[2][16];
  const int nvec = H / N, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const float inv_h = 1.f / (float)H;
  struct Row { P h[VPT], g[VPT], r[VPT]; float rs; };
  float dw[VPT][N];
  P pw[VPT];
  bool live[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    live[i] = v < nvec;
#pragma unroll
    for (int j = 0; j < N; ++j) dw[i][j] = 0.f;
    if (live[i]) pw[i].load_nc(w + v * N);
  }
  auto load = [&](Row& x, int row) {
    const size_t base = (size_t)row * H;
    x.rs = rstd[row];
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = threadIdx.x + i * blockDim.x;
      if (live[i]) {
        x.h[i].load(h + base + v * N);
        x.g[i].load(gy + base + v * N);
        if constexpr (RES) x.r[i].load(gh + base + v * N);
      }
    }
  };
  Row cur, nxt;
  if ((int)blockIdx.x < rows) load(cur, blockIdx.x);
  int buf = 0;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    if (row + (int)gridDim.x < rows) load(nxt, row + gridDim.x);
    const float rs = cur.rs;
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      if (live[i]) {
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const float hh = cur.h[i].f(j) * rs, gg = cur.g[i].f(j);
          dot += gg * pw[i].f(j) * hh;
          dw[i][j] += gg * hh;
        }
      }
    }
    dot = warp_sum(dot);
    if (lane == 0) red[buf][warp] = dot;
    __syncthreads();
    dot = warp_sum(lane < nw ? red[buf][lane] : 0.f) * inv_h;
    buf ^= 1;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = threadIdx.x + i * blockDim.x;
      if (live[i]) {
        P po;
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const float hh = cur.h[i].f(j) * rs;
          const float d = rs * (cur.g[i].f(j) * pw[i].f(j) - hh * dot);
          po.set(j, RES ? cur.r[i].f(j) + d : d);
        }
        po.store(dh + (size_t)row * H + v * N);
      }
    }
    cur = nxt;
  }
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (live[i]) {
      float* o = partial_dw + (size_t)blockIdx.x * H + v * N;
#pragma unroll
      for (int j = 0; j < N; j += 4) *reinterpret_cast<float4*>(o + j) = make_float4(dw[i][j], dw[i][j + 1], dw[i][j + 2], dw[i][j + 3]);
    }
  }
}

// Sum of the blocks' parts of dW, written in the weight's type: 32 columns per block, 32 parts in flight at a time (one thread per
// column that walked all parts took 27 us for 592 parts of 4096 columns).
template <typename T>
static __global__ void __launch_bounds__(256) norm_bwd_reduce_kernel(const float* __restrict__ partial, T* __restrict__ out, int nparts, int H) {
  __shared__ float4 part[32][8];
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3, c = blockIdx.x * 32 + tx * 4;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c < H) {
#pragma unroll 4
    for (int p = ty; p < nparts; p += 32) {
      const float4 v = *reinterpret_cast<const float4*>(partial + (size_t)p * H + c);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
  }
  part[ty][tx] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int col = blockIdx.x * 32 + threadIdx.x;
    float t = 0.f;
#pragma unroll
    for (int y = 0; y < 32; ++y) t += reinterpret_cast<const float*>(part[y])[threadIdx.x];
    if (col < H) out[col] = from_f32<T>(t);
  }
}

template <typename T> static int fn_pick_threads(int H) {
  const int nvec = H / Pack16<T>::N;
  int t = 32;
  while (t < 256 && t * 4 < nvec) t <<= 1;
  return t;
}

#define FN_DISPATCH_DTYPE(dt, ...)                                      \
  switch (dt) {                                                         \
    case kF32: { using T = float; __VA_ARGS__; break; }                 \
    case kBF16: { using T = __nv_bfloat16; __VA_ARGS__; break; }        \
    case kF16: { using T = __half; __VA_ARGS__; break; }                \
    default: nxd_throw("unsupported dtype", __FILE__, __LINE__);        \
  }

void add_rmsnorm_fwd(const void* x, const void* r, const void* w, void* h, void* y, float* rstd, int rows, int H,
                     float eps, int dt, cudaStream_t st) {
  FN_DISPATCH_DTYPE(dt, {
    if (H % Pack16<T>::N) nxd_throw("add_rmsnorm: H must be a multiple of the 16-byte vector width", __FILE__, __LINE__);
    const int th = fn_pick_threads<T>(H);
    auto kernel = H / Pack16<T>::N <= 256 * 4 ? add_rmsnorm_fwd_kernel<T, 4, false> : add_rmsnorm_fwd_kernel<T, 4, true>;
    kernel<<<rows, th, 0, st>>>((const T*)x, (const T*)r, (const T*)w, (T*)h, (T*)y, rstd, H, eps);
  });
  NXD_CUDA_CHECK(cudaGetLastError());
}

int device_sm_count();

// Threads of a block: one packet each up to 512, then two; two to four blocks per SM (one where a thread owns two packets).
static void norm_bwd_shape(int rows, int H, int dt, int& threads, int& vpt, int& grid) {
  const int nvec = H / (dt == kF32 ? 4 : 8);
  threads = std::min(512, (nvec + 31) / 32 * 32);
  vpt = (nvec + threads - 1) / threads;
  const int per_sm = vpt > 1 ? 1 : threads > 256 ? 2 : 4;
  grid = std::min(rows, device_sm_count() * per_sm);
}
int rmsnorm_bwd_num_partials(int rows, int H, int dt) {
  int th, vpt, grid;
  norm_bwd_shape(rows, H, dt, th, vpt, grid);
  return grid;
}

template <bool RES>
static void norm_bwd(const void* gy, const void* gh, const void* h, const void* w, const float* rstd, void* dh, float* partial, void* dw,
                     int rows, int H, int dt, cudaStream_t st) {
  int th, vpt, grid;
  norm_bwd_shape(rows, H, dt, th, vpt, grid);
  FN_DISPATCH_DTYPE(dt, {
    const int nvec = H / Pack16<T>::N;
    if (H % Pack16<T>::N || nvec > 256 * 4) nxd_throw("rmsnorm_bwd: unsupported H", __FILE__, __LINE__);
    if (vpt == 1) norm_bwd_kernel<T, 1, RES><<<grid, th, 0, st>>>((const T*)gy, (const T*)gh, (const T*)h, (const T*)w, rstd, (T*)dh, partial, rows, H);
    else norm_bwd_kernel<T, 2, RES><<<grid, th, 0, st>>>((const T*)gy, (const T*)gh, (const T*)h, (const T*)w, rstd, (T*)dh, partial, rows, H);
    norm_bwd_reduce_kernel<T><<<(H + 31) / 32, 256, 0, st>>>(partial, (T*)dw, grid, H);
  });
  NXD_CUDA_CHECK(cudaGetLastError());
}

void add_rmsnorm_bwd(const void* gy, const void* gh, const void* h, const void* w, const float* rstd, void* dh,
                     float* partial, void* dw, int rows, int H, int dt, cudaStream_t st) {
  norm_bwd<true>(gy, gh, h, w, rstd, dh, partial, dw, rows, H, dt, st);
}
void rmsnorm_bwd(const void* g, const void* x, const void* w, const float* rstd, void* dx, float* partial, void* dw,
                 int rows, int H, int dt, cudaStream_t st) {
  norm_bwd<false>(g, nullptr, x, w, rstd, dx, partial, dw, rows, H, dt, st);
}

}  // namespace nxd

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
#include "sm100_ptx.cuh"

namespace nxd {

// WIDE: rows of more than 256 * MAXV packets; a kernel of its own, since its second loops cost the others registers (bf16: 66 instead
// of 48; 8192 x 5120: 74 us instead of 57).
template <typename T, int MAXV, bool WIDE>
NXD_DEVICE void add_rmsnorm_rows(const T* __restrict__ x, const T* __restrict__ r, const T* __restrict__ w, T* __restrict__ h,
                                 T* __restrict__ y, float* __restrict__ rstd_out, int H, float eps) {
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
      pw.load(w + v * N);
#pragma unroll
      for (int j = 0; j < N; ++j) po.set(j, cache[i].f(j) * rstd * pw.f(j));
      po.store(y + base + v * N);
    }
  }
  for (int v = threadIdx.x + MAXV * blockDim.x; WIDE && v < nvec; v += blockDim.x) {
    P p, pw, po;
    p.load(h + base + v * N);
    pw.load(w + v * N);
#pragma unroll
    for (int j = 0; j < N; ++j) po.set(j, p.f(j) * rstd * pw.f(j));
    po.store(y + base + v * N);
  }
}

template <typename T, int MAXV, bool WIDE>
__global__ void __launch_bounds__(256) add_rmsnorm_fwd_kernel(const T* x, const T* r, const T* w, T* h, T* y, float* rstd_out, int H, float eps) {
  pdl_trigger();
  pdl_wait();
  add_rmsnorm_rows<T, MAXV, WIDE>(x, r, w, h, y, rstd_out, H, eps);
}

// Backward of both norms (RES: with the gradient arriving on the residual path).  Persistent blocks stride over rows; each thread
// owns one or two packets of columns, so its part of dW lives in registers across rows.  Bound by HBM if enough bytes are in flight: whole
// rows come into two stages of shared memory by bulk copies (a row's h, gy and gh are one stage; three or four stages are no faster), and
// the row's sum costs one barrier, behind which the stage is asked for again.  With the loads of the next row in registers instead, the
// blocks per SM were half as many.  Both kernels, bf16 with the residual path, before and now: 8192 x 4096 61.7 and 51.1 us (41 for its
// bytes at the copy rate), 16384 x 4096 111 and 90, 16384 x 1024 45 and 32, 16384 x 8192 171 and 159, 64 x 4096 8.3 and 6.3.
template <typename T, bool RES, int VPT, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT == 1024 ? 1 : VPT == 1 ? 3 : 2) norm_bwd_kernel(const T* gy, const T* gh,
                                                                        const T* h, const T* w,
                                                                        const float* rstd, T* dh,
                                                                        float* partial_dw, int rows, int H) {
  pdl_trigger();                                           // the sum of the parts may take its place; it waits for this grid
  pdl_wait();
  using P = Pack16<T>;
  constexpr int N = P::N;
  extern __shared__ __align__(128) uint8_t ring_raw[];
  __shared__ __align__(16) float red[2][32];
  __shared__ __align__(8) uint64_t full_bar[2];
  const uint32_t ring = smem_u32(ring_raw), full = smem_u32(full_bar);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint32_t row_bytes = (uint32_t)H * sizeof(T), stage_bytes = (RES ? 3 : 2) * row_bytes;
  const float inv_h = 1.f / (float)H;
  auto fetch = [&](unsigned row, int st) {                      // one thread
    const uint32_t dst = ring + st * stage_bytes, bar = full + 8 * st;
    const size_t base = (size_t)row * H;
    mbar_expect_tx(bar, stage_bytes);
    bulk_load(dst, h + base, row_bytes, bar);
    bulk_load(dst + row_bytes, gy + base, row_bytes, bar);
    if constexpr (RES) bulk_load(dst + 2 * row_bytes, gh + base, row_bytes, bar);
  };
  if (threadIdx.x == 0) {
    mbar_init(full, 1);
    mbar_init(full + 8, 1);
    fence_barrier_init();
    fetch(blockIdx.x, 0);                                  // the grid has no more blocks than rows
    if (blockIdx.x + gridDim.x < (unsigned)rows) fetch(blockIdx.x + gridDim.x, 1);
  }
  if (threadIdx.x < 32) red[0][threadIdx.x] = red[1][threadIdx.x] = 0.f;
  float dw[VPT][N];
  P pw[VPT];
  auto at = [&](int i) { return (int)(threadIdx.x + i * blockDim.x) * N; };      // column of this thread's packet i
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
#pragma unroll
    for (int j = 0; j < N; ++j) dw[i][j] = 0.f;
    if (at(i) < H) pw[i].load(w + at(i));
  }
  float rs = rstd[blockIdx.x];
  __syncthreads();
  int st = 0;
  uint32_t ph = 0;
  for (unsigned row = blockIdx.x; row < (unsigned)rows; row += gridDim.x) {
    const float rs_next = row + gridDim.x < (unsigned)rows ? rstd[row + gridDim.x] : 0.f;
    mbar_wait(full + 8 * st, ph);
    P xh[VPT], xg[VPT], xr[VPT];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      if (at(i) < H) {
        const T* src = reinterpret_cast<const T*>(ring_raw + st * stage_bytes) + at(i);
        xh[i].load(src);
        xg[i].load(src + H);
        if constexpr (RES) xr[i].load(src + 2 * H);
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const float hh = xh[i].f(j) * rs, gg = xg[i].f(j);
          dot += gg * pw[i].f(j) * hh;
          dw[i][j] += gg * hh;
        }
      }
    }
    dot = warp_sum(dot);
    if (lane == 0) red[st][warp] = dot;
    __syncthreads();
    if (threadIdx.x == 0 && row + 2 * gridDim.x < (unsigned)rows) fetch(row + 2 * gridDim.x, st);
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    #pragma unroll
    for (int i = 0; i < MAXT / 32; i += 4) {                      // a broadcast read of all warps' sums: shorter than five more shuffles
      const float4 t = *reinterpret_cast<const float4*>(&red[st][i]);
      sum.x += t.x; sum.y += t.y; sum.z += t.z; sum.w += t.w;
    }
    dot = ((sum.x + sum.y) + (sum.z + sum.w)) * inv_h;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      if (at(i) < H) {
        P po;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const float d = rs * (xg[i].f(j) * pw[i].f(j) - (xh[i].f(j) * rs) * dot);
          po.set(j, RES ? xr[i].f(j) + d : d);
        }
        po.store(dh + (size_t)row * H + at(i));
      }
    }
    rs = rs_next;
    st ^= 1;
    if (st == 0) ph ^= 1;
  }
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    if (at(i) < H) {
      float* o = partial_dw + (size_t)blockIdx.x * H + at(i);
#pragma unroll
      for (int j = 0; j < N; j += 4) *reinterpret_cast<float4*>(o + j) = make_float4(dw[i][j], dw[i][j + 1], dw[i][j + 2], dw[i][j + 3]);
    }
  }
}

// Sum of the blocks' parts of dW, written in the weight's type: 32 columns per block, 32 parts in flight at a time (one thread per
// column that walked all parts took 27 us for 592 parts of 4096 columns).
template <typename T>
static __global__ void __launch_bounds__(256) norm_bwd_reduce_kernel(const float* partial, T* out, int nparts, int H) {
  __shared__ float4 part[32][8];
  pdl_wait();
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
    launch_dependent(kernel, rows, th, 0, st, (const T*)x, (const T*)r, (const T*)w, (T*)h, (T*)y, rstd, H, eps);
  });
  NXD_CUDA_CHECK(cudaGetLastError());
}

int device_sm_count();

// Blocks per SM: as registers allow, but a further one only while each block keeps at least four rows (each ends in a part of dW that another
// kernel reads; 1024 x 4096 in blocks of two to three rows 14.4 us, of seven 12.4).  Threads of a block: one packet each, but two
// each between 512 and 768 packets where the rows are enough for two blocks per SM, which then fit (16384 x 6144, without the residual
// path: 104 us, 116 in one block per SM with a packet each).  With fewer rows a packet each is faster: 1024 x 6144 12.3 us, 13.4 with two,
// x 5120 11.2 and 12.5, x 4608 10.3 and 12.3 (with the residual path; caches flushed: 19.5 and 21.5, 19.5 and 21.5, 17.4 and 21.5).
static void norm_bwd_shape(int rows, int H, int dt, int& threads, int& vpt, int& grid) {
  const int size = dt == kF32 ? 4 : 2, nvec = H / (16 / size);
  const int sms = device_sm_count();
  vpt = nvec > 512 && nvec <= 768 && rows >= 8 * sms ? 2 : 1;
  threads = std::max(32, ((nvec + vpt - 1) / vpt + 31) / 32 * 32);
  const int most = std::min(8, (threads > 512 || vpt > 1 ? 1024 : 1536) / threads);
  grid = std::min(rows, sms * std::max(1, std::min(most, rows / (4 * sms))));
}
int rmsnorm_bwd_num_partials(int rows, int H, int dt) {
  int th, vpt, grid;
  norm_bwd_shape(rows, H, dt, th, vpt, grid);
  return grid;
}

template <typename T, bool RES, int VPT, int MAXT>
static void norm_bwd_launch(const void* gy, const void* gh, const void* h, const void* w, const float* rstd, void* dh, float* partial, int rows,
                            int H, int threads, int grid, cudaStream_t st) {
  constexpr int kMost = 6 * 1024 * 16;                     // two stages of three rows of 1024 packets
  NXD_ALLOW_SMEM((norm_bwd_kernel<T, RES, VPT, MAXT>), kMost);
  launch_dependent(norm_bwd_kernel<T, RES, VPT, MAXT>, grid, threads, (size_t)(RES ? 6 : 4) * H * sizeof(T), st,
                   (const T*)gy, (const T*)gh, (const T*)h, (const T*)w, rstd, (T*)dh, partial, rows, H);
}

template <bool RES>
static void norm_bwd(const void* gy, const void* gh, const void* h, const void* w, const float* rstd, void* dh, float* partial, void* dw,
                     int rows, int H, int dt, cudaStream_t st) {
  int th, vpt, grid;
  norm_bwd_shape(rows, H, dt, th, vpt, grid);
  FN_DISPATCH_DTYPE(dt, {
    const int nvec = H / Pack16<T>::N;
    if (H % Pack16<T>::N || nvec > 256 * 4) nxd_throw("rmsnorm_bwd: unsupported H", __FILE__, __LINE__);
    if (vpt == 2) norm_bwd_launch<T, RES, 2, 512>(gy, gh, h, w, rstd, dh, partial, rows, H, th, grid, st);
    else if (th <= 512) norm_bwd_launch<T, RES, 1, 512>(gy, gh, h, w, rstd, dh, partial, rows, H, th, grid, st);
    else norm_bwd_launch<T, RES, 1, 1024>(gy, gh, h, w, rstd, dh, partial, rows, H, th, grid, st);
    launch_dependent(norm_bwd_reduce_kernel<T>, (H + 31) / 32, 256, 0, st, (const float*)partial, (T*)dw, grid, H);
  });
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

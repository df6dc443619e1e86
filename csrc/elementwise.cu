// Hand-written sm_100a elementwise / normalisation / loss kernels.
//   rmsnorm fwd       (reference call site: modules/rms_norm.py:10-33; backward: fused_norm.cu)
//   swiglu  fwd+bwd   (examples/training/llama/modeling_llama_nxd.py:208-219)
//   rope apply        (overrides/transformer_overrides.py:20-32)
//   vocab-parallel cross-entropy stats + backward (parallel_layers/loss_functions.py:12-129)
// All are HBM-bound: 16-byte vector accesses, one pass over the data, fp32 math.
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace nxd {

// =====================================================================================
// RMSNorm forward: one CTA per row, row cached in registers (up to MAXV 16-byte packets/thread)
// =====================================================================================
// EARLY (few rows, where one row's latency is what counts): the weights come to L2 before the wait and into registers with the row.
// A token of 13B 308.3 us, 305.5 so; of a 70B shard 162.8 and 156.9.  With many rows the registers are worth more.
template <typename T, int MAXV, bool EARLY>
__global__ void __launch_bounds__(256) rmsnorm_fwd_kernel(const T* x, const T* w,
                                                          T* y, float* __restrict__ rstd_out, int H,
                                                          float eps) {
  using P = Pack16<T>;
  constexpr int N = P::N;
  __shared__ float red[32];
  pdl_trigger();
  if (EARLY && threadIdx.x == 0) prefetch_l2(w, (uint32_t)H * sizeof(T));
  pdl_wait();
  const int row = blockIdx.x;
  const T* xr = x + (size_t)row * H;
  T* yr = y + (size_t)row * H;
  const int nvec = H / N;
  P cache[MAXV], weights[EARLY ? MAXV : 1];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      cache[i].load(xr + v * N);
      if constexpr (EARLY) weights[i].load(w + v * N);
    }
  }
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    if ((int)(threadIdx.x + i * blockDim.x) < nvec) {
#pragma unroll
      for (int j = 0; j < N; ++j) { const float f = cache[i].f(j); ss += f * f; }
    }
  }
  // tail beyond the register cache (very wide rows): re-read in the second pass
  for (int v = threadIdx.x + MAXV * blockDim.x; v < nvec; v += blockDim.x) {
    P p; p.load(xr + v * N);
#pragma unroll
    for (int j = 0; j < N; ++j) { const float f = p.f(j); ss += f * f; }
  }
  ss = block_sum(ss, red);
  const float rstd = rsqrtf(ss / (float)H + eps);
  if (threadIdx.x == 0) rstd_out[row] = rstd;
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      P pw, po;
      if constexpr (EARLY) pw = weights[i];
      else pw.load(w + v * N);
#pragma unroll
      for (int j = 0; j < N; ++j) po.set(j, cache[i].f(j) * rstd * pw.f(j));
      po.store(yr + v * N);
    }
  }
  for (int v = threadIdx.x + MAXV * blockDim.x; v < nvec; v += blockDim.x) {
    P p, pw, po; p.load(xr + v * N); pw.load(w + v * N);
#pragma unroll
    for (int j = 0; j < N; ++j) po.set(j, p.f(j) * rstd * pw.f(j));
    po.store(yr + v * N);
  }
}

// =====================================================================================
// SwiGLU: out[t, i] = silu(gu[t, i]) * gu[t, I + i]
// =====================================================================================
template <typename T>
__global__ void __launch_bounds__(256) swiglu_fwd_kernel(const T* gu, T* out, size_t rows, int I) {
  using P = Pack16<T>;
  constexpr int N = P::N;
  pdl_trigger();
  pdl_wait();
  const int vec_per_row = I / N;
  const size_t total = rows * (size_t)vec_per_row;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
    const size_t r = idx / vec_per_row;
    const int c = (int)(idx % vec_per_row) * N;
    P pg, pu, po;
    pg.load(gu + r * 2 * I + c);
    pu.load(gu + r * 2 * I + I + c);
#pragma unroll
    for (int j = 0; j < N; ++j) po.set(j, silu_mul(pg.f(j), pu.f(j)));
    po.store(out + r * I + c);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) swiglu_bwd_kernel(const T* go, const T* gu,
                                                         T* dgu, size_t rows, int I) {
  pdl_trigger();
  pdl_wait();
  using P = Pack16<T>;
  constexpr int N = P::N;
  const int vec_per_row = I / N;
  const size_t total = rows * (size_t)vec_per_row;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
    const size_t r = idx / vec_per_row;
    const int c = (int)(idx % vec_per_row) * N;
    P pg, pu, pd, og, ou;
    pg.load(gu + r * 2 * I + c);
    pu.load(gu + r * 2 * I + I + c);
    pd.load(go + r * I + c);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const float g = pg.f(j), u = pu.f(j), d = pd.f(j);
      const float sig = 1.f / (1.f + __expf(-g));
      const float silu = g * sig;
      og.set(j, d * u * (sig + silu * (1.f - sig)));
      ou.set(j, d * silu);
    }
    og.store(dgu + r * 2 * I + c);
    ou.store(dgu + r * 2 * I + I + c);
  }
}

// =====================================================================================
// RoPE (rotate-half).  x: [B,S,H,D] with arbitrary B/S/H strides (D contiguous) → out contiguous.
// sign=+1 forward, -1 backward (inverse rotation).  One thread: 8 elements of each half.
// =====================================================================================
// One packet of each half of a head: (a, b) -> (a cos - b sin, b cos + a sin); sign -1 rotates back.
template <typename T>
__device__ __forceinline__ void rotate(const Pack16<T>& p1, const Pack16<T>& p2, const float* __restrict__ cr, const float* __restrict__ sr,
                                       float sign, Pack16<T>& o1, Pack16<T>& o2) {
#pragma unroll
  for (int j = 0; j < Pack16<T>::N; ++j) {
    const float cs = cr[j], sn = sr[j] * sign;
    const float a = p1.f(j), bb = p2.f(j);
    o1.set(j, a * cs - bb * sn);
    o2.set(j, bb * cs + a * sn);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) rope_kernel(const T* x, T* out,
                                                   const float* cos_t, const float* sin_t,
                                                   int B, int S, int Hh, int D, long sb, long ss, long sh, float sign) {
  pdl_trigger();
  pdl_wait();
  using P = Pack16<T>;
  constexpr int N = P::N;
  const int half = D / 2;
  const int vec_per_head = half / N;
  const size_t total = (size_t)B * S * Hh * vec_per_head;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
    const int c = (int)(idx % vec_per_head) * N;
    size_t t = idx / vec_per_head;
    const int h = (int)(t % Hh); t /= Hh;
    const int s = (int)(t % S);
    const int b = (int)(t / S);
    const T* src = x + b * sb + s * ss + h * sh;
    T* dst = out + (((size_t)b * S + s) * Hh + h) * D;
    P p1, p2, o1, o2;
    p1.load(src + c);
    p2.load(src + half + c);
    const float* cr = cos_t + (size_t)s * half + c;
    const float* sr = sin_t + (size_t)s * half + c;
    rotate(p1, p2, cr, sr, sign, o1, o2);
    o1.store(dst + c);
    o2.store(dst + half + c);
  }
}

// Rotation of q and k out of the fused projection [S, B, (H + 2 K) D], and back: the gradients of q and k rotated back, that of v
// copied, into one fused gradient.  Bound by memory; one block per token row, the two halves of a head are 16-byte packets of one
// thread.  With the caches flushed, 2048 tokens x (32 + 2 x 32) heads of 128 take 18.5 us forward and 29.6 back (10.3 and 15.4 at the
// copy rate); two rotations each way and a concatenation took 23.6 and 37.9.  4 x 1024 x (32 + 2 x 8): 20.5 and 30.9, were 25.6 and 138.
template <typename T>
__global__ void __launch_bounds__(256) rope_qkv_fwd_kernel(const T* x, T* q, T* k,
                                                           const float* cos_t, const float* sin_t, int B, int H,
                                                           int K, int D, float sign) {
  pdl_trigger();
  pdl_wait();
  using P = Pack16<T>;
  constexpr int N = P::N;
  const int half = D / 2, per = half / N, s = blockIdx.x / B, S = gridDim.x / B;
  const size_t to = (size_t)(blockIdx.x - s * B) * S + s;
  const T* row = x + (size_t)blockIdx.x * (H + 2 * K) * D;
  for (int i = threadIdx.x; i < (H + K) * per; i += 256) {
    const int h = i / per, c = (i - h * per) * N;
    T* dst = h < H ? q + (to * H + h) * D : k + (to * K + h - H) * D;
    P p1, p2, o1, o2;
    p1.load(row + (size_t)h * D + c);
    p2.load(row + (size_t)h * D + half + c);
    const float* cr = cos_t + (size_t)s * half + c;
    const float* sr = sin_t + (size_t)s * half + c;
    rotate(p1, p2, cr, sr, sign, o1, o2);
    o1.store(dst + c);
    o2.store(dst + half + c);
  }
}

// A gradient [B, S, heads, D] and its strides over batch, position and head.
struct RopeGrad { const void* p; long sb, ss, sh; };
template <typename T>
__global__ void __launch_bounds__(256) rope_qkv_bwd_kernel(const RopeGrad gq, const RopeGrad gk, const RopeGrad gv, T* out,
                                                           const float* cos_t, const float* sin_t, int B, int H,
                                                           int K, int D, float sign) {
  pdl_trigger();
  pdl_wait();
  using P = Pack16<T>;
  constexpr int N = P::N;
  const int half = D / 2, per = half / N, s = blockIdx.x / B, b = blockIdx.x - s * B;
  T* row = out + (size_t)blockIdx.x * (H + 2 * K) * D;
  for (int i = threadIdx.x; i < (H + 2 * K) * per; i += 256) {
    const int h = i / per, c = (i - h * per) * N;
    const RopeGrad& g = h < H ? gq : h < H + K ? gk : gv;
    const int hh = h < H ? h : h < H + K ? h - H : h - H - K;
    const T* src = (const T*)g.p + b * g.sb + s * g.ss + hh * g.sh;
    P p1, p2, o1, o2;
    p1.load(src + c);
    p2.load(src + half + c);
    if (h < H + K) {
      const float* cr = cos_t + (size_t)s * half + c;
      const float* sr = sin_t + (size_t)s * half + c;
      rotate(p1, p2, cr, sr, sign, o1, o2);
    } else {
      o1 = p1; o2 = p2;
    }
    o1.store(row + (size_t)h * D + c);
    o2.store(row + (size_t)h * D + half + c);
  }
}

// Prompts of served models: q rotated into a tensor of its own, k rotated and v copied into rows 0..S-1 of the caches, which the attention
// then reads.  One block per token row, as above.  1000 tokens, 40 + 2 x 40 heads of 128: two rotations and two copies took 12 and 16 us a
// layer; a prompt through two layers got 23 us shorter.
template <typename T>
__global__ void __launch_bounds__(256) prefill_rope_kv_kernel(const RopeGrad gq, const RopeGrad gk, const RopeGrad gv, T* q_out, T* kc, T* vc,
                                                              long c_sb, long c_ss, long c_sh, const float* cos_t, const float* sin_t, int B,
                                                              int S, int H, int K, int D) {
  using P = Pack16<T>;
  constexpr int N = P::N;
  pdl_trigger();
  pdl_wait();
  const int half = D / 2, per = half / N, s = blockIdx.x / B, b = blockIdx.x - s * B;
  for (int i = threadIdx.x; i < (H + 2 * K) * per; i += 256) {
    const int h = i / per, c = (i - h * per) * N;
    const RopeGrad& g = h < H ? gq : h < H + K ? gk : gv;
    const int hh = h < H ? h : h < H + K ? h - H : h - H - K;
    const T* src = (const T*)g.p + b * g.sb + s * g.ss + hh * g.sh;
    T* dst = h < H ? q_out + (((size_t)b * S + s) * H + hh) * D : (h < H + K ? kc : vc) + b * c_sb + s * c_ss + hh * c_sh;
    P p1, p2, o1, o2;
    p1.load(src + c);
    p2.load(src + half + c);
    if (h < H + K) {
      rotate(p1, p2, cos_t + (size_t)s * half + c, sin_t + (size_t)s * half + c, 1.f, o1, o2);
    } else {
      o1 = p1; o2 = p2;
    }
    o1.store(dst + c);
    o2.store(dst + half + c);
  }
}

// =====================================================================================
// Cross-entropy statistics: per row (max, sum exp(x-max), target logit if owned, sum x).
// One CTA per row; online softmax per thread then block merge.
// =====================================================================================
template <typename T>
__global__ void __launch_bounds__(256) ce_stats_kernel(const T* __restrict__ logits, const int64_t* __restrict__ target,
                                                       float* __restrict__ stats, int V, int vocab_start, int vec) {
  using P = Pack16<T>;
  constexpr int N = P::N;
  __shared__ float red[32];
  const int row = blockIdx.x;
  const T* xr = logits + (size_t)row * V;
  float m = -INFINITY, s = 0.f, sx = 0.f;
  const int nvec = vec ? V / N : 0;                 // rows of another alignment: element by element
  // fmaxf passes NaN by, so behind nothing but masked columns and NaN the maximum is still -inf: the terms are then taken against 0,
  // where a masked column adds 0 and NaN adds NaN, and the sum is NaN in the end wherever one stood
  auto take = [&](const P& p) {
    float lm = m;
#pragma unroll
    for (int j = 0; j < N; ++j) lm = fmaxf(lm, p.f(j));
    const float ref = lm == -INFINITY ? 0.f : lm;
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) { const float f = p.f(j); acc += __expf(f - ref); sx += f; }
    s = s * __expf(m - ref) + acc;
    m = lm;
  };
  int v = threadIdx.x;
  constexpr int U = 4;                              // packets in flight per thread
  for (; v + (U - 1) * (int)blockDim.x < nvec; v += U * blockDim.x) {
    P p[U];
#pragma unroll
    for (int u = 0; u < U; ++u) p[u].load(xr + (size_t)(v + u * blockDim.x) * N);
#pragma unroll
    for (int u = 0; u < U; ++u) take(p[u]);
  }
  for (; v < nvec; v += blockDim.x) { P p; p.load(xr + (size_t)v * N); take(p); }
  for (int c = nvec * N + threadIdx.x; c < V; c += blockDim.x) {  // ragged tail
    const float f = to_f32<T>(xr[c]);
    const float nm = fmaxf(m, f), ref = nm == -INFINITY ? 0.f : nm;
    s = s * __expf(m - ref) + __expf(f - ref);
    m = nm; sx += f;
  }
  const float gm = block_max(m, red);
  const float contrib = s * __expf(m - (gm == -INFINITY ? 0.f : gm));      // m = -inf: 0, or NaN
  const float gs = block_sum(contrib, red);
  const float gsx = block_sum(sx, red);
  if (threadIdx.x == 0) {
    const long local = (long)target[row] - vocab_start;
    const float tl = (local >= 0 && local < V) ? to_f32<T>(xr[local]) : 0.f;
    float* o = stats + (size_t)row * 4;
    o[0] = gm; o[1] = gs; o[2] = tl; o[3] = gsx;
  }
}

// largest element of packets (NaN passed by, as by fmaxf)
template <int U> NXD_DEVICE float packets_max(const Pack16<float> (&p)[U]) {
  float m = -INFINITY;
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int j = 0; j < 4; ++j) m = fmaxf(m, p[u].f(j));
  return m;
}
template <typename T, int U> NXD_DEVICE float packets_max(const Pack16<T> (&p)[U]) {
  using T2 = typename std::conditional<std::is_same<T, __half>::value, __half2, __nv_bfloat162>::type;
  T2 m[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) m[j] = reinterpret_cast<const T2*>(p[0].v)[j];
#pragma unroll
  for (int u = 1; u < U; ++u)
#pragma unroll
    for (int j = 0; j < 4; ++j) m[j] = __hmax2(m[j], reinterpret_cast<const T2*>(p[u].v)[j]);
  const T2 a = __hmax2(__hmax2(m[0], m[1]), __hmax2(m[2], m[3]));
  return fmaxf(fmaxf(to_f32<T>(a.x), to_f32<T>(a.y)), -INFINITY);       // NaN only: -inf
}

// Loss and log-normaliser of rows that hold the whole vocabulary: the pass of ce_stats_kernel, finished in the same launch.  One block per
// row.  A thread takes its packets in groups of four that are loaded together, the last group too (what lies beyond the row reads as
// -inf), and corrects its sum once per group; sums and products two per instruction.  Bound by HBM and the exponential unit (busy for two
// thirds of the time).  4096 x 32000, bf16: 44 us (40 at the copy rate), ce_stats_kernel 49 and three launches of 1.9 to 3.1 behind it;
// a ring of bulk copies under persistent blocks took 49 too.
template <typename T, int THREADS>
__global__ void __launch_bounds__(THREADS, 2048 / THREADS) ce_loss_kernel(const T* logits, const int64_t* target,
                                                                           float* lse, float* loss, int V, int vec) {
  pdl_trigger();
  pdl_wait();
  using P = Pack16<T>;
  constexpr int N = P::N, U = 4;                // packets in flight per thread
  __shared__ float red[32];
  const int row = blockIdx.x;
  const T* xr = logits + (size_t)row * V;
  float m = -INFINITY, s = 0.f;
  const int nvec = vec ? V / N : 0;                 // rows of another alignment: element by element
  const uint64_t log2e = pack2(1.4426950408889634f, 1.4426950408889634f);
  for (int v = threadIdx.x; v < nvec; v += U * THREADS) {
    P p[U];
    const int n = (nvec - v + THREADS - 1) / THREADS;             // live packets, if less than U
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u < n) p[u].load(xr + (size_t)(v + u * THREADS) * N);
      else
#pragma unroll
        for (int j = 0; j < N; ++j) p[u].set(j, -INFINITY);      // no maximum, and nothing in a sum of exponentials
    }
    const float lm = fmaxf(m, packets_max(p));
    const float ref = lm == -INFINITY ? 0.f : lm;
    const uint64_t nref = pack2(-ref, -ref);
    uint64_t acc = 0ull;
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int j = 0; j < N; j += 2) {
        float a, b;
        unpack2(mul2(add2(pack2(p[u].f(j), p[u].f(j + 1)), nref), log2e), a, b);
        acc = add2(acc, pack2(ex2(a), ex2(b)));
      }
    }
    float a, b;
    unpack2(acc, a, b);
    s = s * __expf(m - ref) + (a + b);
    m = lm;
  }
  for (int c = nvec * N + threadIdx.x; c < V; c += THREADS) {  // ragged tail
    const float f = to_f32<T>(xr[c]);
    const float nm = fmaxf(m, f), ref = nm == -INFINITY ? 0.f : nm;
    s = s * __expf(m - ref) + __expf(f - ref);
    m = nm;
  }
  const float gm = block_max(m, red);
  const float contrib = s * __expf(m - (gm == -INFINITY ? 0.f : gm));      // m = -inf: 0, or NaN
  const float gs = block_sum(contrib, red);
  if (threadIdx.x == 0) {
    const long local = (long)target[row];
    const float tl = (local >= 0 && local < V) ? to_f32<T>(xr[local]) : 0.f;
    const float l = gm + (float)log((double)gs);           // the 32-bit logarithm of this build is an approximation
    lse[row] = l;
    loss[row] = l - tl;
  }
}

template <typename T>
__global__ void __launch_bounds__(256) ce_bwd_kernel(const T* logits, const int64_t* target,
                                                     const float* lse, const float* gout,
                                                     T* grad, int V, int vocab_start, float smoothing,
                                                     float inv_vocab, int vec) {
  pdl_trigger();
  pdl_wait();
  using P = Pack16<T>;
  constexpr int N = P::N;
  const int row = gridDim.x - 1 - blockIdx.x;       // the rows that the statistics read last are the ones still in L2
  const T* xr = logits + (size_t)row * V;
  T* gr = grad + (size_t)row * V;
  const float l = lse[row], g = gout[row];
  long local = (long)target[row] - vocab_start;
  if (local < 0 || local >= V) local = -1;          // no column of this shard
  const float sm_term = smoothing * inv_vocab;
  const int nvec = vec ? V / N : 0;
#pragma unroll 4
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    P p, o;
    *reinterpret_cast<uint4*>(p.v) = __ldcs(reinterpret_cast<const uint4*>(xr + v * N));
    const int at = (int)(local - (long)v * N);      // of the target within this packet, if in 0..N-1
#pragma unroll
    for (int j = 0; j < N; ++j) {
      float d = __expf(p.f(j) - l) - sm_term;
      if (j == at) d -= (1.f - smoothing);
      o.set(j, d * g);
    }
    __stcs(reinterpret_cast<uint4*>(gr + v * N), *reinterpret_cast<const uint4*>(o.v));
  }
  for (int c = nvec * N + threadIdx.x; c < V; c += blockDim.x) {
    float d = __expf(to_f32<T>(xr[c]) - l) - sm_term;
    if ((long)c == local) d -= (1.f - smoothing);
    gr[c] = from_f32<T>(d * g);
  }
}

// The mean of a causal language model's losses around those two passes: what the labels say of each row (s, b) of [S, B] logits, the mean of the
// rows that count, and the gradient that the mean gives each of them.  Seventeen elementwise launches and their nodes did this: 1960 us a step of
// the two-layer model whose time is the host's, 1830 with these.
__global__ void __launch_bounds__(256) lm_targets_kernel(const int64_t* labels, long sb, long ss, int64_t* target, float* mask, int S, int B, int shift) {
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x * 256 + threadIdx.x;
  if (r >= S * B) return;
  const int s = r / B + shift, b = r % B;
  const int64_t t = s < S ? labels[b * sb + s * ss] : -100;
  target[r] = t == -100 ? 0 : t;                // rows that do not count are taken along, as target 0 times 0
  mask[r] = t == -100 ? 0.f : 1.f;
}

// one block: sum(loss * mask) / max(sum(mask), 1) and its divisor; the sum in 64 bits
__global__ void __launch_bounds__(1024) lm_mean_kernel(const float* loss, const float* mask, float* mean, float* divisor, int rows) {
  pdl_trigger();
  pdl_wait();
  double sum = 0.;
  int count = 0;
#pragma unroll 4
  for (int r = threadIdx.x; r < rows; r += 1024) {
    const float m = mask[r];
    sum += (double)(loss[r] * m);
    count += m != 0.f;
  }
  __shared__ double sums[32];
  __shared__ int counts[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    count += __shfl_xor_sync(0xffffffffu, count, o);
  }
  if (threadIdx.x % 32 == 0) { sums[threadIdx.x / 32] = sum; counts[threadIdx.x / 32] = count; }
  __syncthreads();
  if (threadIdx.x) return;
  for (int w = 1; w < 32; ++w) { sum += sums[w]; count += counts[w]; }
  const float n = (float)max(count, 1);
  *mean = (float)sum / n;
  *divisor = n;
}

__global__ void __launch_bounds__(256) lm_row_grads_kernel(const float* gout, const float* divisor, const float* mask, float* grads, int rows) {
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x * 256 + threadIdx.x;
  if (r < rows) grads[r] = *gout / *divisor * mask[r];
}

// ---------------------------------------------------------------- launchers
template <typename T> static int pick_threads(int H) {
  const int nvec = H / Pack16<T>::N;
  int t = 32;
  while (t < 256 && t * 4 < nvec) t <<= 1;   // aim for <= 4 packets / thread
  return t;
}

#define DISPATCH_DTYPE(dt, ...)                                         \
  switch (dt) {                                                         \
    case kF32: { using T = float; __VA_ARGS__; break; }                 \
    case kBF16: { using T = __nv_bfloat16; __VA_ARGS__; break; }        \
    case kF16: { using T = __half; __VA_ARGS__; break; }                \
    default: nxd_throw("unsupported dtype", __FILE__, __LINE__);        \
  }

int device_sm_count();
static int num_sms() { return device_sm_count(); }

void rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, int rows, int H, float eps, int dt, cudaStream_t st) {
  DISPATCH_DTYPE(dt, {
    if (H % Pack16<T>::N) nxd_throw("rmsnorm: H must be a multiple of the 16-byte vector width", __FILE__, __LINE__);
    const int th = pick_threads<T>(H);
    auto kernel = rows <= 64 ? rmsnorm_fwd_kernel<T, 4, true> : rmsnorm_fwd_kernel<T, 4, false>;
    launch_dependent(kernel, rows, th, 0, st, (const T*)x, (const T*)w, (T*)y, rstd, H, eps);
  });
  NXD_CUDA_CHECK(cudaGetLastError());
}

void swiglu_fwd(const void* gu, void* out, long rows, int I, int dt, cudaStream_t st) {
  DISPATCH_DTYPE(dt, {
    const size_t total = (size_t)rows * (I / Pack16<T>::N);
    const int grid = (int)min((size_t)num_sms() * 16, (total + 255) / 256);
    launch_dependent(swiglu_fwd_kernel<T>, max(grid, 1), 256, 0, st, (const T*)gu, (T*)out, (size_t)rows, I);
  });
  NXD_CUDA_CHECK(cudaGetLastError());
}

void swiglu_bwd(const void* go, const void* gu, void* dgu, long rows, int I, int dt, cudaStream_t st) {
  DISPATCH_DTYPE(dt, {
    const size_t total = (size_t)rows * (I / Pack16<T>::N);
    const int grid = (int)min((size_t)num_sms() * 16, (total + 255) / 256);
    launch_dependent(swiglu_bwd_kernel<T>, max(grid, 1), 256, 0, st, (const T*)go, (const T*)gu, (T*)dgu, (size_t)rows, I);
  });
  NXD_CUDA_CHECK(cudaGetLastError());
}

// any even D (partial rotary dims such as GPT-NeoX-20B's 24 of 96): one element pair per thread
template <typename T>
__global__ void __launch_bounds__(256) rope_scalar_kernel(const T* __restrict__ x, T* __restrict__ out,
                                                          const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                                          int B, int S, int Hh, int D, long sb, long ss, long sh, float sign) {
  const int half = D / 2;
  const size_t total = (size_t)B * S * Hh * half;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
    const int c = (int)(idx % half);
    size_t t = idx / half;
    const int h = (int)(t % Hh); t /= Hh;
    const int s = (int)(t % S);
    const int b = (int)(t / S);
    const T* src = x + b * sb + s * ss + h * sh;
    T* dst = out + (((size_t)b * S + s) * Hh + h) * D;
    const float cs = cos_t[(size_t)s * half + c], sn = sin_t[(size_t)s * half + c] * sign;
    const float a = to_f32<T>(src[c]), bb = to_f32<T>(src[half + c]);
    dst[c] = from_f32<T>(a * cs - bb * sn);
    dst[half + c] = from_f32<T>(bb * cs + a * sn);
  }
}

void rope_apply(const void* x, void* out, const float* cos_t, const float* sin_t, int B, int S, int Hh, int D, long sb,
                long ss, long sh, float sign, int dt, cudaStream_t st) {
  DISPATCH_DTYPE(dt, {
    if (D % 2) nxd_throw("rope: D must be even", __FILE__, __LINE__);
    if ((D / 2) % Pack16<T>::N || ((uintptr_t)x % 16) || (sb * sizeof(T)) % 16 || (ss * sizeof(T)) % 16 || (sh * sizeof(T)) % 16) {
      const size_t total = (size_t)B * S * Hh * (D / 2);
      const int grid = (int)min((size_t)num_sms() * 16, (total + 255) / 256);
      rope_scalar_kernel<T><<<max(grid, 1), 256, 0, st>>>((const T*)x, (T*)out, cos_t, sin_t, B, S, Hh, D, sb, ss, sh, sign);
      NXD_CUDA_CHECK(cudaGetLastError());
      return;
    }
    const size_t total = (size_t)B * S * Hh * ((D / 2) / Pack16<T>::N);
    const int grid = (int)min((size_t)num_sms() * 16, (total + 255) / 256);
    launch_dependent(rope_kernel<T>, max(grid, 1), 256, 0, st, (const T*)x, (T*)out, cos_t, sin_t, B, S, Hh, D, sb, ss, sh, sign);
  });
  NXD_CUDA_CHECK(cudaGetLastError());
}

void rope_qkv_fwd(const void* x, void* q, void* k, const float* cos_t, const float* sin_t, int S, int B, int H, int K, int D, int dt,
                  cudaStream_t st) {
  if (S * B == 0) return;
  DISPATCH_DTYPE(dt, {
    launch_dependent(rope_qkv_fwd_kernel<T>, S * B, 256, 0, st, (const T*)x, (T*)q, (T*)k, cos_t, sin_t, B, H, K, D, 1.0f);
  });
  NXD_CUDA_CHECK(cudaGetLastError());
}
// strides[i] = (batch, position, head) of gq, gk, gv
void rope_qkv_bwd(const void* gq, const void* gk, const void* gv, const long (*strides)[3], void* out, const float* cos_t, const float* sin_t,
                  int S, int B, int H, int K, int D, int dt, cudaStream_t st) {
  if (S * B == 0) return;
  const RopeGrad g[3] = {{gq, strides[0][0], strides[0][1], strides[0][2]}, {gk, strides[1][0], strides[1][1], strides[1][2]},
                         {gv, strides[2][0], strides[2][1], strides[2][2]}};
  DISPATCH_DTYPE(dt, {
    launch_dependent(rope_qkv_bwd_kernel<T>, S * B, 256, 0, st, g[0], g[1], g[2], (T*)out, cos_t, sin_t, B, H, K, D, -1.0f);
  });
  NXD_CUDA_CHECK(cudaGetLastError());
}

// strides of q, k, v: batch, position, head; caches [B, L, K, D] with one set of strides
void prefill_rope_kv(const void* q, const void* k, const void* v, const long (*strides)[3], void* q_out, void* kc, void* vc, const long* cs,
                     const float* cos_t, const float* sin_t, int B, int S, int H, int K, int D, int dt, cudaStream_t st) {
  if (S * B == 0) return;
  const RopeGrad g[3] = {{q, strides[0][0], strides[0][1], strides[0][2]}, {k, strides[1][0], strides[1][1], strides[1][2]},
                         {v, strides[2][0], strides[2][1], strides[2][2]}};
  DISPATCH_DTYPE(dt, {
    launch_dependent(prefill_rope_kv_kernel<T>, S * B, 256, 0, st, g[0], g[1], g[2], (T*)q_out, (T*)kc, (T*)vc, cs[0], cs[1], cs[2], cos_t, sin_t,
                     B, S, H, K, D);
  });
}

void ce_stats(const void* logits, const int64_t* target, float* stats, int rows, int V, int vocab_start, int dt,
              cudaStream_t st) {
  DISPATCH_DTYPE(dt, {
    const int vec = (uintptr_t)logits % 16 == 0 && V % Pack16<T>::N == 0;
    ce_stats_kernel<T><<<rows, 256, 0, st>>>((const T*)logits, target, stats, V, vocab_start, vec);
  });
  NXD_CUDA_CHECK(cudaGetLastError());
}

// Threads: 256, but 512 where rows are long (4000 x 128256: 151 us, 155 with 256; 4096 x 4000: 25, 14 with 256) or too few to fill the
// SMs (128 x 32000: 5.2, 6.5 with 256).
void ce_loss(const void* logits, const int64_t* target, float* lse, float* loss, int rows, int V, int dt, cudaStream_t st) {
  DISPATCH_DTYPE(dt, {
    const int vec = (uintptr_t)logits % 16 == 0 && V % Pack16<T>::N == 0;
    auto go = [&](auto kernel, int threads) { launch_dependent(kernel, rows, threads, 0, st, (const T*)logits, target, lse, loss, V, vec); };
    if ((long)V * sizeof(T) >= 128 << 10 || rows <= 2 * num_sms()) go(ce_loss_kernel<T, 512>, 512);
    else go(ce_loss_kernel<T, 256>, 256);
  });
  NXD_CUDA_CHECK(cudaGetLastError());
}

void lm_targets(const int64_t* labels, long sb, long ss, int64_t* target, float* mask, int S, int B, bool shift, cudaStream_t st) {
  launch_dependent(lm_targets_kernel, (S * B + 255) / 256, 256, 0, st, labels, sb, ss, target, mask, S, B, (int)shift);
  NXD_CUDA_CHECK(cudaGetLastError());
}
void lm_mean(const float* loss, const float* mask, float* mean, float* divisor, int rows, cudaStream_t st) {
  launch_dependent(lm_mean_kernel, 1, 1024, 0, st, loss, mask, mean, divisor, rows);
  NXD_CUDA_CHECK(cudaGetLastError());
}
void lm_row_grads(const float* gout, const float* divisor, const float* mask, float* grads, int rows, cudaStream_t st) {
  launch_dependent(lm_row_grads_kernel, (rows + 255) / 256, 256, 0, st, gout, divisor, mask, grads, rows);
  NXD_CUDA_CHECK(cudaGetLastError());
}

void ce_backward(const void* logits, const int64_t* target, const float* lse, const float* gout, void* grad, int rows,
                 int V, int vocab_start, float smoothing, int vocab, int dt, cudaStream_t st) {
  DISPATCH_DTYPE(dt, {
    const int vec = ((uintptr_t)logits | (uintptr_t)grad) % 16 == 0 && V % Pack16<T>::N == 0;
    launch_dependent(ce_bwd_kernel<T>, rows, 256, 0, st, (const T*)logits, target, lse, gout, (T*)grad, V, vocab_start, smoothing,
                                           1.f / (float)vocab, vec);
  });
  NXD_CUDA_CHECK(cudaGetLastError());
}

}  // namespace nxd

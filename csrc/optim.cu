// Multi-tensor optimizer kernels: one launch covers a whole list of tensors through a chunk table
// passed by value in kernel parameters (no per-tensor launches, no host sync).
//   multi_tensor_sq_norm : Σ‖t‖² → atomicAdd into a device fp32 scalar   (grads.py:41-189)
//   multi_tensor_scale   : t *= *scale (device scalar; clip coefficient) (grads.py:238-256)
//   fused_adamw          : fp32 master/moment update + optional bf16 model copy
//                          (utils/adamw_fp32_optim_params.py:91-155)
#include <algorithm>

#include <cuda.h>

#include "common.cuh"
#include "kernels.h"
#include "sm100_ptx.cuh"

namespace nxd {

constexpr int kMaxTensors = 48;
constexpr long kChunk = 4096;   // elements of a chunk
constexpr int kBlocksPerSm = 6;

// Up to 48 tensors of a launch, cut into chunks; blocks stride over all chunks, so that the launch ends evenly whatever the sizes
// (640 blocks of 65536 elements per launch were 4.3 per SM, five on some).  Squared norm of 0.67 G fp32 elements: 492 -> 397 us
// (6.7 TB/s).
template <int DEPTH> struct ChunkTable {
  void* ptr[DEPTH][kMaxTensors];
  long numel[kMaxTensors];
  long first[kMaxTensors + 1];  // first chunk of each tensor
  int tensors;
};

// tensor of chunk c
template <int DEPTH>
NXD_DEVICE int tensor_of(const ChunkTable<DEPTH>& tab, long c) {
  int lo = 0, hi = tab.tensors - 1;
  while (lo < hi) {
    const int mid = (lo + hi) / 2;
    if (tab.first[mid + 1] <= c) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// calls f(tensor, first element, elements) for every chunk of this block
template <int DEPTH, typename F>
NXD_DEVICE void each_chunk(const ChunkTable<DEPTH>& tab, F&& f) {
  int t = tensor_of(tab, blockIdx.x);
  for (long c = blockIdx.x; c < tab.first[tab.tensors]; c += gridDim.x) {
    while (tab.first[t + 1] <= c) ++t;
    const long base = (c - tab.first[t]) * kChunk;
    f(t, base, min(tab.numel[t] - base, kChunk));
  }
}

template <typename T>
__global__ void __launch_bounds__(256) sq_norm_kernel(const __grid_constant__ ChunkTable<1> tab, float* __restrict__ out) {
  __shared__ float red[32];
  float s = 0.f;
  each_chunk(tab, [&](int t, long base, long n) {
    const T* p = (const T*)tab.ptr[0][t] + base;
    constexpr int N = Pack16<T>::N;
    long i0 = 0;
    if (((uintptr_t)p % 16) == 0) {
      const long nv = n / N;
#pragma unroll 4
      for (long v = threadIdx.x; v < nv; v += 256) {
        Pack16<T> k; k.load_nc(p + v * N);
#pragma unroll
        for (int j = 0; j < N; ++j) { const float f = k.f(j); s += f * f; }
      }
      i0 = nv * N;
    }
    for (long i = i0 + threadIdx.x; i < n; i += 256) { const float f = to_f32<T>(p[i]); s += f * f; }
  });
  s = block_sum(s, red);
  if (threadIdx.x == 0) atomicAdd(out, s);
}

// the norm of a squared norm and what clipping to max_norm multiplies the gradients by: five launches of one element, 25 us of the host's time in a step
// of two layers that lasts 1750
__global__ void clip_kernel(const float* sq, float max_norm, float* norm, float* coeff) {
  float n;
  asm("sqrt.rn.f32 %0, %1;" : "=f"(n) : "f"(*sq));                   // a subnormal is not taken for zero
  const float c = __frcp_rn(n + 1e-6f) * max_norm;
  *norm = n;
  *coeff = c > 1.f ? 1.f : c;                    // NaN stays
}

template <typename T>
__global__ void __launch_bounds__(256) scale_kernel(const __grid_constant__ ChunkTable<1> tab, const float* __restrict__ scale) {
  const float sc = *scale;
  each_chunk(tab, [&](int t, long base, long n) {
    T* p = (T*)tab.ptr[0][t] + base;
    constexpr int N = Pack16<T>::N;
    long i0 = 0;
    if (((uintptr_t)p % 16) == 0) {
      const long nv = n / N;
#pragma unroll 4
      for (long v = threadIdx.x; v < nv; v += 256) {
        Pack16<T> k; k.load(p + v * N);
#pragma unroll
        for (int j = 0; j < N; ++j) k.set(j, k.f(j) * sc);
        k.store(p + v * N);
      }
      i0 = nv * N;
    }
    for (long i = i0 + threadIdx.x; i < n; i += 256) p[i] = from_f32<T>(to_f32<T>(p[i]) * sc);
  });
}

// buffer = gradient, or += it, in fp32: a 16-bit gradient that autograd delivers into the optimizer's buffer.  Bound by HBM: four
// elements per access, so that a warp's stores are whole lines, and eight accesses in flight per thread.  32000 x 4096 bf16: 137 us (5.7 TB/s), added 204; as copy_ 351.
template <typename G, bool ADD>
__global__ void __launch_bounds__(256) grad_to_buffer_kernel(const G* __restrict__ g, float* __restrict__ buf, long n) {
  constexpr int U = 8;
  const long quads = n / 4, step = (long)gridDim.x * 256;
  const uint2* g4 = reinterpret_cast<const uint2*>(g);
  float4* b4 = reinterpret_cast<float4*>(buf);
  auto put = [&](const uint2& raw, long v) {
    const G* x = reinterpret_cast<const G*>(&raw);
    float4 y = make_float4(to_f32<G>(x[0]), to_f32<G>(x[1]), to_f32<G>(x[2]), to_f32<G>(x[3]));
    if (ADD) { const float4 b = b4[v]; y.x += b.x; y.y += b.y; y.z += b.z; y.w += b.w; }
    b4[v] = y;
  };
  long v = (long)blockIdx.x * 256 + threadIdx.x;
  for (; v + (U - 1) * step < quads; v += U * step) {
    uint2 x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = __ldg(g4 + v + u * step);
#pragma unroll
    for (int u = 0; u < U; ++u) put(x[u], v + u * step);
  }
  for (; v < quads; v += step) put(__ldg(g4 + v), v);
  for (long i = quads * 4 + (long)blockIdx.x * 256 + threadIdx.x; i < n; i += step) buf[i] = ADD ? buf[i] + to_f32<G>(g[i]) : to_f32<G>(g[i]);
}

// One update rule covers both AdamW forms:
//   p = (p * decay_pre - step_size * m / (sqrt(v * vscale) + eps)) * decay_post
// torch form : step_size = lr/bc1, vscale = 1/bc2, decay_pre = 1 - lr*wd, decay_post = 1
// HF form    : step_size = lr*sqrt(bc2)/bc1, vscale = 1, decay_pre = 1, decay_post = 1 - lr*wd
//              (reference utils/adamw_fp32_optim_params.py:130-155: eps added before bias correction, decay applied last)
struct AdamRule {
  float step_size, beta1, beta2, eps, decay_pre, decay_post, vscale;
  NXD_DEVICE float operator()(float gr, float& m, float& v, float p) const {
    m = beta1 * m + (1.f - beta1) * gr;
    v = beta2 * v + (1.f - beta2) * gr * gr;
    return (p * decay_pre - step_size * m / (sqrtf(v * vscale) + eps)) * decay_post;
  }
};

constexpr int kAdamThreads = 512;
constexpr int kAdamStages = 3;
constexpr int kAdamStage = 5 * (int)kChunk * 4 - (int)kChunk * 2;       // p, g, m, v and a 16-bit copy: 72 KB
constexpr int kAdamSmem = kAdamStages * kAdamStage + 64;

// One chunk in global memory: four elements per access where fp32 arrays are 16-byte aligned and 16-bit ones 8-byte, else one.
template <typename G, typename L, bool HAS_LOW>
NXD_DEVICE void adam_in_place(float* p, const G* g, float* m, float* v, L* low, int n, const AdamRule& rule, float gs) {
  int i0 = 0;
  if ((((uintptr_t)p | (uintptr_t)m | (uintptr_t)v) % 16) == 0 && (uintptr_t)g % (4 * sizeof(G)) == 0 && (!HAS_LOW || (uintptr_t)low % (4 * sizeof(L)) == 0)) {
    i0 = n / 4 * 4;
#pragma unroll 2
    for (int i = threadIdx.x * 4; i < i0; i += blockDim.x * 4) {
      float4 pp = *reinterpret_cast<const float4*>(p + i), mm = *reinterpret_cast<const float4*>(m + i), vv = *reinterpret_cast<const float4*>(v + i);
      float gg[4];
      if constexpr (sizeof(G) == 4) {
        const float4 t4 = *reinterpret_cast<const float4*>(g + i);
        gg[0] = t4.x; gg[1] = t4.y; gg[2] = t4.z; gg[3] = t4.w;
      } else {
        const uint2 raw = *reinterpret_cast<const uint2*>(g + i);
        const G* h = reinterpret_cast<const G*>(&raw);
#pragma unroll
        for (int j = 0; j < 4; ++j) gg[j] = to_f32<G>(h[j]);
      }
      float* pa = &pp.x; float* ma = &mm.x; float* va = &vv.x;
#pragma unroll
      for (int j = 0; j < 4; ++j) pa[j] = rule(gg[j] * gs, ma[j], va[j], pa[j]);
      *reinterpret_cast<float4*>(p + i) = pp;
      *reinterpret_cast<float4*>(m + i) = mm;
      *reinterpret_cast<float4*>(v + i) = vv;
      if constexpr (HAS_LOW) {
        if constexpr (sizeof(L) == 4) {
          *reinterpret_cast<float4*>(low + i) = pp;
        } else {
          uint2 raw; L* h = reinterpret_cast<L*>(&raw);
#pragma unroll
          for (int j = 0; j < 4; ++j) h[j] = from_f32<L>(pa[j]);
          *reinterpret_cast<uint2*>(low + i) = raw;
        }
      }
    }
  }
  for (int i = i0 + threadIdx.x; i < n; i += blockDim.x) {
    float mi = m[i], vi = v[i];
    const float pi = rule(to_f32<G>(g[i]) * gs, mi, vi, p[i]);
    m[i] = mi; v[i] = vi; p[i] = pi;
    if constexpr (HAS_LOW) low[i] = from_f32<L>(pi);
  }
}

// Tensors that the bulk copies of adamw_kernel cannot take (an array that is not 16-byte aligned: slices).  64 tensors of 1 M elements,
// 16-bit arrays 8-byte aligned / all arrays off by one element: 337 us (5.6 TB/s) and 435; element by element on the bulk kernel 730 and 804.
template <typename G, typename L, bool HAS_LOW>
__global__ void __launch_bounds__(256) adamw_direct_kernel(const __grid_constant__ ChunkTable<5> tab, const AdamRule rule,
                                                           const float* __restrict__ grad_scale) {
  const float gs = grad_scale ? *grad_scale : 1.f;
  each_chunk(tab, [&](int t, long base, long n) {
    adam_in_place<G, L, HAS_LOW>((float*)tab.ptr[0][t] + base, (const G*)tab.ptr[1][t] + base, (float*)tab.ptr[2][t] + base,
                                 (float*)tab.ptr[3][t] + base, HAS_LOW ? (L*)tab.ptr[4][t] + base : nullptr, (int)n, rule, gs);
  });
}

// Bound by HBM: 16 + 14 bytes per element with fp32 gradients and a bf16 copy: four streams in, four out.  Whole chunks travel as bulk
// copies of 16 KB through a ring in shared memory, updated in place there: a stream's bytes reach a DRAM page together.  0.67 G
// elements: 3.09 ms (6.5 TB/s); with 16-byte accesses per thread 3.70 (5.4), however the blocks were cut.  Chunks that are shorter
// (the ends of tensors) are updated in global memory.
template <typename G, typename L, bool HAS_LOW>
__global__ void __launch_bounds__(kAdamThreads, 1) adamw_kernel(const __grid_constant__ ChunkTable<5> tab, const AdamRule rule,
                                                                const float* __restrict__ grad_scale) {
  extern __shared__ __align__(128) uint8_t adam_smem[];
  const uint32_t base = smem_u32(adam_smem), bars = base + kAdamStages * kAdamStage;
  const float gs = grad_scale ? *grad_scale : 1.f;
  const long total = tab.first[tab.tensors];
  const int tid = threadIdx.x;
  if (tid == 0) {
    for (int i = 0; i < kAdamStages; ++i) mbar_init(bars + 8 * i, 1);
    fence_barrier_init();
  }
  __syncthreads();
  struct Chunk { float *p, *m, *v; const G* g; L* low; int n; bool bulk; };
  int t_at = tensor_of(tab, blockIdx.x), t_load = t_at;      // chunks are visited in ascending order
  auto find = [&](long c, int& t) {
    while (tab.first[t + 1] <= c) ++t;
    const long off = (c - tab.first[t]) * kChunk;
    Chunk k;
    k.p = (float*)tab.ptr[0][t] + off; k.g = (const G*)tab.ptr[1][t] + off;
    k.m = (float*)tab.ptr[2][t] + off; k.v = (float*)tab.ptr[3][t] + off;
    k.low = HAS_LOW ? (L*)tab.ptr[4][t] + off : nullptr;
    k.n = (int)min(tab.numel[t] - off, kChunk);
    k.bulk = k.n == kChunk;                        // the arrays are 16-byte aligned
    return k;
  };
  constexpr uint32_t F = (uint32_t)kChunk * 4, GB = (uint32_t)kChunk * sizeof(G), LB = (uint32_t)kChunk * sizeof(L);
  static_assert(4 * kChunk * 4 + kChunk * 2 == kAdamStage && sizeof(L) <= 4, "stage layout");
  // an fp32 copy equals p and is stored from there
  auto load = [&](const Chunk& k, int st) {        // thread 0
    const uint32_t s = base + st * kAdamStage, bar = bars + 8 * st;
    mbar_expect_tx(bar, 3 * F + GB);
    auto copy = [&](uint32_t dst, const void* src, uint32_t bytes) {
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                   ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
    };
    copy(s, k.p, F); copy(s + F, k.m, F); copy(s + 2 * F, k.v, F); copy(s + 3 * F, k.g, GB);
  };
  auto store = [&](void* dst, uint32_t src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
  };
  long next = blockIdx.x;                          // next chunk to ask for (thread 0)
  auto load_next = [&](int st) {
    if (next < total) {
      const Chunk k = find(next, t_load);
      if (k.bulk) load(k, st);
    }
    next += gridDim.x;
  };
  if (tid == 0) { load_next(0); load_next(1); }
  uint32_t phases = 0;                             // parity of each stage's barrier
  int st = 0;
  for (long c = blockIdx.x; c < total; c += gridDim.x) {
    const Chunk k = find(c, t_at);
    if (k.bulk) {
      mbar_wait(bars + 8 * st, (phases >> st) & 1u);
      phases ^= 1u << st;
      uint8_t* s = adam_smem + st * kAdamStage;
      float4* sp = reinterpret_cast<float4*>(s);
      float4* sm = reinterpret_cast<float4*>(s + F);
      float4* sv = reinterpret_cast<float4*>(s + 2 * F);
#pragma unroll
      for (int q = tid; q < (int)kChunk / 4; q += kAdamThreads) {
        float4 pp = sp[q], mm = sm[q], vv = sv[q];
        float gg[4];
        if constexpr (sizeof(G) == 4) {
          const float4 t4 = reinterpret_cast<const float4*>(s + 3 * F)[q];
          gg[0] = t4.x; gg[1] = t4.y; gg[2] = t4.z; gg[3] = t4.w;
        } else {
          const uint2 raw = reinterpret_cast<const uint2*>(s + 3 * F)[q];
          const G* h = reinterpret_cast<const G*>(&raw);
#pragma unroll
          for (int j = 0; j < 4; ++j) gg[j] = to_f32<G>(h[j]);
        }
        float* pa = &pp.x; float* ma = &mm.x; float* va = &vv.x;
#pragma unroll
        for (int j = 0; j < 4; ++j) pa[j] = rule(gg[j] * gs, ma[j], va[j], pa[j]);
        sp[q] = pp; sm[q] = mm; sv[q] = vv;
        if constexpr (HAS_LOW && sizeof(L) == 2) {
          uint2 raw; L* h = reinterpret_cast<L*>(&raw);
#pragma unroll
          for (int j = 0; j < 4; ++j) h[j] = from_f32<L>(pa[j]);
          reinterpret_cast<uint2*>(s + 4 * F)[q] = raw;
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    } else {
      adam_in_place<G, L, HAS_LOW>(k.p, k.g, k.m, k.v, k.low, k.n, rule, gs);
    }
    __syncthreads();
    if (tid == 0) {
      if (k.bulk) {
        const uint32_t s = base + st * kAdamStage;
        store(k.p, s, F); store(k.m, s + F, F); store(k.v, s + 2 * F, F);
        if constexpr (HAS_LOW) store(k.low, sizeof(L) == 2 ? s + 4 * F : s, LB);
      }
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");      // the stage before has left: it takes the chunk after the next
      load_next((st + 2) % kAdamStages);
    }
    st = (st + 1) % kAdamStages;
  }
  if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

int device_sm_count();

// launches once per 48 tensors
template <int DEPTH, typename Launch>
static void run_tables(const std::vector<TensorRef>* lists, int blocks_per_sm, Launch&& launch) {
  ChunkTable<DEPTH> tab;
  tab.tensors = 0;
  tab.first[0] = 0;
  auto flush = [&]() {
    const long chunks = tab.first[tab.tensors];
    if (chunks > 0) launch(tab, (int)std::min<long>(chunks, (long)device_sm_count() * blocks_per_sm));
    tab.tensors = 0;
  };
  for (size_t t = 0; t < lists[0].size(); ++t) {
    const long numel = lists[0][t].numel;
    if (numel == 0) continue;
    if (tab.tensors == kMaxTensors) flush();
    const int slot = tab.tensors++;
    for (int d = 0; d < DEPTH; ++d) tab.ptr[d][slot] = lists[d].empty() ? nullptr : lists[d][t].ptr;
    tab.numel[slot] = numel;
    tab.first[slot + 1] = tab.first[slot] + (numel + kChunk - 1) / kChunk;
  }
  flush();
}

void clip_coefficient(const float* sq, float max_norm, float* norm, float* coeff, cudaStream_t st) {
  clip_kernel<<<1, 1, 0, st>>>(sq, max_norm, norm, coeff);
  NXD_CUDA_CHECK(cudaGetLastError());
}

void multi_tensor_sq_norm(const std::vector<TensorRef>& ts, int dt, float* out, cudaStream_t st) {
  const std::vector<TensorRef> lists[1] = {ts};
  run_tables<1>(lists, kBlocksPerSm, [&](const ChunkTable<1>& tab, int nb) {
    switch (dt) {
      case kF32: sq_norm_kernel<float><<<nb, 256, 0, st>>>(tab, out); break;
      case kBF16: sq_norm_kernel<__nv_bfloat16><<<nb, 256, 0, st>>>(tab, out); break;
      case kF16: sq_norm_kernel<__half><<<nb, 256, 0, st>>>(tab, out); break;
      default: nxd_throw("bad dtype", __FILE__, __LINE__);
    }
  });
  NXD_CUDA_CHECK(cudaGetLastError());
}

void multi_tensor_scale(const std::vector<TensorRef>& ts, int dt, const float* scale, cudaStream_t st) {
  const std::vector<TensorRef> lists[1] = {ts};
  run_tables<1>(lists, kBlocksPerSm, [&](const ChunkTable<1>& tab, int nb) {
    switch (dt) {
      case kF32: scale_kernel<float><<<nb, 256, 0, st>>>(tab, scale); break;
      case kBF16: scale_kernel<__nv_bfloat16><<<nb, 256, 0, st>>>(tab, scale); break;
      case kF16: scale_kernel<__half><<<nb, 256, 0, st>>>(tab, scale); break;
      default: nxd_throw("bad dtype", __FILE__, __LINE__);
    }
  });
  NXD_CUDA_CHECK(cudaGetLastError());
}

void grad_to_buffer(const void* grad, int dt, float* buffer, long n, bool add, cudaStream_t st) {
  if (n == 0) return;
  const int grid = (int)std::min<long>((n / 4 + 255) / 256 + 1, (long)device_sm_count() * 8);
#define NXD_G2B(G)                                                                                        \
  do {                                                                                                    \
    if (add) grad_to_buffer_kernel<G, true><<<grid, 256, 0, st>>>((const G*)grad, buffer, n);             \
    else grad_to_buffer_kernel<G, false><<<grid, 256, 0, st>>>((const G*)grad, buffer, n);                \
  } while (0)
  if (dt == kBF16) NXD_G2B(__nv_bfloat16);
  else if (dt == kF16) NXD_G2B(__half);
  else nxd_throw("grad_to_buffer: 16-bit gradients", __FILE__, __LINE__);
#undef NXD_G2B
  NXD_CUDA_CHECK(cudaGetLastError());
}

void fused_adamw(const std::vector<TensorRef>& p, const std::vector<TensorRef>& g, const std::vector<TensorRef>& m,
                 const std::vector<TensorRef>& v, const std::vector<TensorRef>& lowp, int gdt, int ldt, float lr,
                 float beta1, float beta2, float eps, float wd, float bc1, float bc2, const float* grad_scale,
                 int hf_form, cudaStream_t st) {
  const std::vector<TensorRef>* lists[5] = {&p, &g, &m, &v, &lowp};
  const bool has_low = !lowp.empty();
  AdamRule rule{hf_form ? lr * sqrtf(bc2) / bc1 : lr / bc1, beta1, beta2, eps, hf_form ? 1.f : 1.f - lr * wd, hf_form ? 1.f - lr * wd : 1.f,
                hf_form ? 1.f : 1.f / bc2};
  std::vector<TensorRef> parts[2][5];              // 16-byte aligned throughout, others
  for (int d = 0; d < 5; ++d) parts[0][d].reserve(lists[d]->size());
  for (size_t t = 0; t < p.size(); ++t) {
    uintptr_t bits = 0;
    for (const auto* l : lists) if (!l->empty()) bits |= (uintptr_t)(*l)[t].ptr;
    for (int d = 0; d < 5; ++d) if (!lists[d]->empty()) parts[bits % 16 != 0][d].push_back((*lists[d])[t]);
  }
  for (int direct = 0; direct < 2; ++direct) run_tables<5>(parts[direct], direct ? kBlocksPerSm : 1, [&](const ChunkTable<5>& tab, int nb) {
#define LAUNCH(G, L, HL)                                                                                                     \
  do {                                                                                                                       \
    if (direct) { adamw_direct_kernel<G, L, HL><<<nb, 256, 0, st>>>(tab, rule, grad_scale); break; }                         \
    NXD_ALLOW_SMEM((adamw_kernel<G, L, HL>), kAdamSmem);                                                                     \
    adamw_kernel<G, L, HL><<<nb, kAdamThreads, kAdamSmem, st>>>(tab, rule, grad_scale);                                      \
  } while (0)
    if (gdt == kF32) {
      if (!has_low) LAUNCH(float, float, false);
      else if (ldt == kBF16) LAUNCH(float, __nv_bfloat16, true);
      else if (ldt == kF16) LAUNCH(float, __half, true);
      else LAUNCH(float, float, true);
    } else if (gdt == kBF16) {
      if (!has_low) LAUNCH(__nv_bfloat16, float, false);
      else if (ldt == kBF16) LAUNCH(__nv_bfloat16, __nv_bfloat16, true);
      else if (ldt == kF16) LAUNCH(__nv_bfloat16, __half, true);
      else LAUNCH(__nv_bfloat16, float, true);
    } else {
      if (!has_low) LAUNCH(__half, float, false);
      else if (ldt == kF16) LAUNCH(__half, __half, true);
      else if (ldt == kBF16) LAUNCH(__half, __nv_bfloat16, true);
      else LAUNCH(__half, float, true);
    }
#undef LAUNCH
  });
  NXD_CUDA_CHECK(cudaGetLastError());
}

}  // namespace nxd

// RMSNorm forward / backward (LLaMA and Gemma "1+w" flavours) with an optional fused residual add.
//
// Forward: one CTA (128 threads) per token row; the row stays in registers between the
// sum-of-squares pass and the scale pass, so HBM traffic is exactly read-x (+read-residual) and
// write-y (+write-residual).  Backward: persistent CTAs walk rows, produce dx and keep the weight
// gradient in registers; per-CTA partials are reduced by a second tiny kernel (colsum.cuh).
// Replaces the eager fp32-upcast RMSNorm of the reference (modules/mlp.py:425-467).
#include <atomic>

#include "colsum.cuh"

namespace {

constexpr int kThreads = 128;

template <typename T, bool kResidual, int kMaxVec>
__global__ void __launch_bounds__(kThreads) rmsnorm_fwd_kernel(const T* __restrict__ x, const T* __restrict__ res_in,
                                                               const T* __restrict__ w, T* __restrict__ y,
                                                               T* __restrict__ res_out, float* __restrict__ rstd_out,
                                                               int H, float eps, float w_offset) {
  __shared__ float red[32];
  constexpr int V = 8;
  const int64_t row = blockIdx.x;
  const int nvec = H / V;
  rb::pdl_trigger();  // successors may start launching (and prefetching weights) while this kernel still waits below
  rb::pdl_wait();
  const rb::Pack<T, V>* xr = reinterpret_cast<const rb::Pack<T, V>*>(x + row * H);
  const rb::Pack<T, V>* rr = kResidual ? reinterpret_cast<const rb::Pack<T, V>*>(res_in + row * H) : nullptr;
  float vals[kMaxVec][V];
  float ss = 0.f;
#pragma unroll
  for (int it = 0; it < kMaxVec; ++it) {
    const int i = threadIdx.x + it * kThreads;
    if (i < nvec) {
      rb::Pack<T, V> a = xr[i];
      if constexpr (kResidual) {
        rb::Pack<T, V> b = rr[i];
        rb::Pack<T, V> o;
#pragma unroll
        for (int k = 0; k < V; ++k) {
          // round the residual stream to T first so the normalised value matches what is stored
          o.v[k] = rb::from_f<T>(rb::to_f(a.v[k]) + rb::to_f(b.v[k]));
          vals[it][k] = rb::to_f(o.v[k]);
        }
        reinterpret_cast<rb::Pack<T, V>*>(res_out + row * H)[i] = o;
      } else {
#pragma unroll
        for (int k = 0; k < V; ++k) vals[it][k] = rb::to_f(a.v[k]);
      }
#pragma unroll
      for (int k = 0; k < V; ++k) ss = fmaf(vals[it][k], vals[it][k], ss);
    }
  }
  ss = rb::block_reduce<false>(ss, red);
  const float rstd = rsqrtf(ss / (float)H + eps);
  if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
  const rb::Pack<T, V>* wr = reinterpret_cast<const rb::Pack<T, V>*>(w);
#pragma unroll
  for (int it = 0; it < kMaxVec; ++it) {
    const int i = threadIdx.x + it * kThreads;
    if (i < nvec) {
      rb::Pack<T, V> ww = wr[i], o;
#pragma unroll
      for (int k = 0; k < V; ++k) o.v[k] = rb::from_f<T>(vals[it][k] * rstd * (rb::to_f(ww.v[k]) + w_offset));
      reinterpret_cast<rb::Pack<T, V>*>(y + row * H)[i] = o;
    }
  }
}

// The same for few rows, as a generation step has: nothing but latency.  A thread has one piece of the row and asks for all that it reads at once ; with
// four pieces of 4096 columns a thread, and the weight asked for behind the reduction, 16 rows took 3.05 us back to back, now 1.82, and 3.4 us more than now in a
// generation step, where nothing of it is in a cache.  Up to two rows an SM it is never behind (bf16 with residual, the general kernel / this one: 296 rows x 768
// 1.64 / 1.56 us, x 4096 4.98 / 3.33, x 8192 8.55 / 5.62; 592 x 4096 6.31 / 4.96 but x 8192 9.19 / 10.21; 1184 x 4096 6.89 / 7.63).
template <typename T, bool kResidual>
__global__ void __launch_bounds__(1024) rmsnorm_few_kernel(const T* __restrict__ x, const T* __restrict__ res_in, const T* __restrict__ w, T* __restrict__ y,
                                                           T* __restrict__ res_out, float* __restrict__ rstd_out, int H, float eps, float w_offset) {
  __shared__ float red[32];
  constexpr int V = 8;
  using Vec = rb::Pack<T, V>;
  const int64_t at = (int64_t)blockIdx.x * (H / V) + threadIdx.x;
  const bool mine = threadIdx.x < H / V;
  rb::pdl_trigger();
  rb::pdl_wait();
  Vec a{}, b{}, ww{};
  if (mine) {
    a = reinterpret_cast<const Vec*>(x)[at];
    if constexpr (kResidual) b = reinterpret_cast<const Vec*>(res_in)[at];
    ww = reinterpret_cast<const Vec*>(w)[threadIdx.x];
  }
  float v[V], ss = 0.f;
#pragma unroll
  for (int k = 0; k < V; ++k) {
    if constexpr (kResidual) a.v[k] = rb::from_f<T>(rb::to_f(a.v[k]) + rb::to_f(b.v[k]));   // rounded first, so that the norm is that of what is stored
    v[k] = rb::to_f(a.v[k]);
    ss = fmaf(v[k], v[k], ss);
  }
  if constexpr (kResidual) {
    if (mine) reinterpret_cast<Vec*>(res_out)[at] = a;
  }
  ss = rb::block_reduce<false>(ss, red);
  const float rstd = rsqrtf(ss / (float)H + eps);
  if (threadIdx.x == 0 && rstd_out) rstd_out[blockIdx.x] = rstd;
#pragma unroll
  for (int k = 0; k < V; ++k) b.v[k] = rb::from_f<T>(v[k] * rstd * (rb::to_f(ww.v[k]) + w_offset));
  if (mine) reinterpret_cast<Vec*>(y)[at] = b;
}

// dx = rstd * (g - xhat * mean(g*xhat)) (+ dres),  g = dy * (w + off);  dw += dy * xhat
//
// Bound by HBM: x, dy (and the gradient arriving on the residual stream, `dres`) in, dx out.  A row is one reduction deep, so a CTA that
// loads, reduces and stores row after row leaves the memory idle for most of each row (20480 x 4096 bf16 with dres: 220 us, 3.0 TB/s; with
// one row prefetched into registers 192 us).  Every thread therefore keeps the pieces of kStages rows in flight with cp.async, into
// shared memory only it reads back (no barrier, no wait on another thread), and the reduction takes one barrier (two alternating sets of
// warp sums).  The rings of an SM hold 192 KB (16-bit rows of up to 1024 columns: 96 KB, four CTAs), a third of it for dres.
// A thread's pieces of a row are 16 bytes, TB pieces apart, so that a warp's copies cover whole lines (with 8 consecutive fp32 elements a thread every copy
// touched half of twice as many sectors: 12000 x 2048 fp32 with dres 94 us, 65 this way).
template <typename T, int TB, int NV> struct RmsBwd {
  static constexpr int kStageBytes = 3 * NV * TB * 16;
  static constexpr int kStages = kStageBytes > 48 * 1024 ? 2 : 4;
  static constexpr int kSmem = kStages * kStageBytes;
  static constexpr int kFit = 200 * 1024 / kSmem, kCtas = kFit > 4 ? 4 : kFit;   // 4: the partial sums have 4 rows per SM
};

RB_DEVICE void cp_async16(uint32_t dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
RB_DEVICE void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> RB_DEVICE void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <typename T, int TB, int NV>
__global__ void __launch_bounds__(TB, RmsBwd<T, TB, NV>::kCtas)
    rmsnorm_bwd_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ dy, const float* __restrict__ rstd, T* __restrict__ dx,
                       float* __restrict__ dw_partial, int64_t T_rows, int H, float w_offset, const T* __restrict__ dres) {
  using C = RmsBwd<T, TB, NV>;
  constexpr int V = 16 / sizeof(T), kWarps = TB / 32;
  using Vec = rb::Pack<T, V>;
  extern __shared__ uint4 ring[];       // [kStages][3 operands][NV][TB]
  __shared__ float red[2][kWarps];
  const int nvec = H / V, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float inv_h = 1.f / (float)H;
  float dw[NV][V];
  Vec wv[NV];
#pragma unroll
  for (int it = 0; it < NV; ++it) {
    const int i = threadIdx.x + it * TB;
#pragma unroll
    for (int k = 0; k < V; ++k) dw[it][k] = 0.f;
    if (i < nvec) wv[it] = reinterpret_cast<const Vec*>(w)[i];
  }
  auto slot = [&](int st, int op, int it) { return ring + ((st * 3 + op) * NV + it) * TB + threadIdx.x; };
  auto fetch = [&](int64_t row, int st) {
    if (row < T_rows) {
#pragma unroll
      for (int it = 0; it < NV; ++it) {
        const int i = threadIdx.x + it * TB;
        if (i < nvec) {
          const int64_t at = row * H + (int64_t)i * V;
          cp_async16((uint32_t)__cvta_generic_to_shared(slot(st, 0, it)), x + at);
          cp_async16((uint32_t)__cvta_generic_to_shared(slot(st, 1, it)), dy + at);
          if (dres != nullptr) cp_async16((uint32_t)__cvta_generic_to_shared(slot(st, 2, it)), dres + at);
        }
      }
    }
    cp_async_commit();                  // (an empty group past the end keeps the count)
  };
  auto take = [&](int st, int op, int it) {
    Vec v;
    *reinterpret_cast<uint4*>(&v) = *slot(st, op, it);
    return v;
  };
#pragma unroll
  for (int st = 0; st < C::kStages; ++st) fetch(blockIdx.x + (int64_t)st * gridDim.x, st);
  int par = 0, st = 0;
  float rs_next = blockIdx.x < T_rows ? rstd[blockIdx.x] : 0.f;
  for (int64_t row = blockIdx.x; row < T_rows; row += gridDim.x, par ^= 1) {
    const float rs = rs_next;
    if (row + gridDim.x < T_rows) rs_next = rstd[row + gridDim.x];
    cp_async_wait<C::kStages - 1>();
    Vec a[NV], d[NV], e[NV];
    float dot = 0.f;
#pragma unroll
    for (int it = 0; it < NV; ++it) {
      if (threadIdx.x + it * TB < nvec) {
        a[it] = take(st, 0, it);
        d[it] = take(st, 1, it);
        if (dres != nullptr) e[it] = take(st, 2, it);
#pragma unroll
        for (int k = 0; k < V; ++k) {
          const float xh = rb::to_f(a[it].v[k]) * rs, dyk = rb::to_f(d[it].v[k]);
          dw[it][k] = fmaf(dyk, xh, dw[it][k]);
          dot = fmaf(dyk * (rb::to_f(wv[it].v[k]) + w_offset), xh, dot);
        }
      }
    }
    dot = rb::warp_sum(dot);
    if (lane == 0) red[par][warp] = dot;
    __syncthreads();     // (the other set is rewritten only behind the next row's barrier)
    fetch(row + (int64_t)C::kStages * gridDim.x, st);
    st = st + 1 == C::kStages ? 0 : st + 1;
    dot = 0.f;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) dot += red[par][k];
    dot *= inv_h;
#pragma unroll
    for (int it = 0; it < NV; ++it) {
      const int i = threadIdx.x + it * TB;
      if (i < nvec) {
        Vec o;
#pragma unroll
        for (int k = 0; k < V; ++k) {
          const float xh = rb::to_f(a[it].v[k]) * rs, g = rb::to_f(d[it].v[k]) * (rb::to_f(wv[it].v[k]) + w_offset);
          float v = rs * (g - xh * dot);
          if (dres != nullptr) v += rb::to_f(e[it].v[k]);
          o.v[k] = rb::from_f<T>(v);
        }
        reinterpret_cast<Vec*>(dx + row * H)[i] = o;
      }
    }
  }
#pragma unroll
  for (int it = 0; it < NV; ++it) {
    const int i = threadIdx.x + it * TB;
    if (i < nvec) {
#pragma unroll
      for (int k = 0; k < V; k += 4)
        *reinterpret_cast<float4*>(dw_partial + (int64_t)blockIdx.x * H + i * V + k) = make_float4(dw[it][k], dw[it][k + 1], dw[it][k + 2], dw[it][k + 3]);
    }
  }
}

template <typename T, int TB, int NV>
int launch_rmsnorm_bwd(const void* x, const void* w, const void* dy, const float* rstd, void* dx, float* dw_partial, void* dw, int64_t rows, int H,
                       float w_offset, const void* dres, cudaStream_t s) {
  using C = RmsBwd<T, TB, NV>;
  auto kern = rmsnorm_bwd_kernel<T, TB, NV>;
  static std::atomic<uint64_t> opted_in{0};          // the attribute is the kernel's on one device: a bit per device
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -2;
  if (dev >= 64 || !(opted_in.load() >> dev & 1)) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem) != cudaSuccess) return -2;
    if (dev < 64) opted_in.fetch_or(1ull << dev);
  }
  const int64_t ctas = (int64_t)rb::kNumSMs * C::kCtas;
  const int grid = (int)(rows < ctas ? rows : ctas);
  kern<<<grid, TB, C::kSmem, s>>>((const T*)x, (const T*)w, (const T*)dy, rstd, (T*)dx, dw_partial, rows, H, w_offset, (const T*)dres);
  if (cudaGetLastError() != cudaSuccess) return -3;
  rb::launch_colsum<T>(dw_partial, dw, grid, H, s);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace

extern "C" {

// dt: 0 fp32, 1 bf16, 2 fp16.  H must be a multiple of 8 and <= 8192.
int rb_rmsnorm_fwd(const void* x, const void* res_in, const void* w, void* y, void* res_out, float* rstd, int64_t rows,
                   int H, float eps, float w_offset, int dt, cudaStream_t s) {
  if (rows == 0) return 0;
  if (H % 8 != 0 || H > kThreads * 8 * 8) return -1;
#define RB_FEW(T, R) \
  return rb::launch_pdl(rmsnorm_few_kernel<T, R>, dim3((unsigned)rows), dim3(RB_CEIL_DIV(H, 256) * 32), 0, s, (const T*)x, (const T*)res_in, (const T*)w, (T*)y, \
                        (T*)res_out, rstd, H, eps, w_offset) == cudaSuccess ? 0 : -3
  if (rows <= 2 * rb::kNumSMs) {
    if (dt == 0) { if (res_in) RB_FEW(float, true); RB_FEW(float, false); }
    if (dt == 1) { if (res_in) RB_FEW(__nv_bfloat16, true); RB_FEW(__nv_bfloat16, false); }
    if (dt == 2) { if (res_in) RB_FEW(__half, true); RB_FEW(__half, false); }
    return -1;
  }
#undef RB_FEW
#define RB_L2(T, NV)                                                                                               \
  if (res_in) rb::launch_pdl(rmsnorm_fwd_kernel<T, true, NV>, dim3((unsigned)rows), dim3(kThreads), 0, s,                \
      (const T*)x, (const T*)res_in, (const T*)w, (T*)y, (T*)res_out, rstd, H, eps, w_offset);                         \
  else rb::launch_pdl(rmsnorm_fwd_kernel<T, false, NV>, dim3((unsigned)rows), dim3(kThreads), 0, s, (const T*)x,       \
                      (const T*)nullptr, (const T*)w, (T*)y, (T*)nullptr, rstd, H, eps, w_offset);
#define RB_L(T)                                                            \
  { const int nv = RB_CEIL_DIV(H, kThreads * 8);                            \
    if (nv <= 1) { RB_L2(T, 1) } else if (nv <= 2) { RB_L2(T, 2) } else if (nv <= 4) { RB_L2(T, 4) } else { RB_L2(T, 8) } }
  if (dt == 0) { RB_L(float) } else if (dt == 1) { RB_L(__nv_bfloat16) } else if (dt == 2) { RB_L(__half) } else return -1;
#undef RB_L
#undef RB_L2
  return 0;
}

int rb_rmsnorm_bwd_num_partials() { return rb::kNumSMs * 4; }

int rb_rmsnorm_bwd(const void* x, const void* w, const void* dy, const float* rstd, void* dx, float* dw_partial,
                   void* dw, int64_t rows, int H, float w_offset, int dt, const void* dres, cudaStream_t s) {
  if (rows == 0) return 0;
  if (H % 8 != 0 || H > kThreads * 8 * 8) return -1;
  // 128 threads up to 1024 columns, 256 beyond; NV: pieces of 8 columns a thread, in fp32 twice as many of 4
#define RB_L2(T, TB, NV) return launch_rmsnorm_bwd<T, TB, NV * (int)sizeof(T) / 2>(x, w, dy, rstd, dx, dw_partial, dw, rows, H, w_offset, dres, s)
#define RB_L(T)                                                                                                       \
  { if (H <= 1024) RB_L2(T, 128, 1); if (H <= 2048) RB_L2(T, 256, 1); if (H <= 4096) RB_L2(T, 256, 2); RB_L2(T, 256, 4); }
  if (dt == 0) { RB_L(float) } else if (dt == 1) { RB_L(__nv_bfloat16) } else if (dt == 2) { RB_L(__half) } else return -1;
#undef RB_L
#undef RB_L2
}

}  // extern "C"

// Pieces shared by the tcgen05 attention kernels: parameters, bounded waits, packing, the soft cap.
#pragma once
#include "gemm_common.cuh"

namespace rb {

struct AttnParams {
  const int* cu_seqlens;  // [B + 1]
  void* out;              // [T, nq, D]
  float* lse;             // [nq, T]
  int64_t out_ld;         // elements between consecutive tokens of `out`
  int T, nq, nkv;
  float scale;
  int causal;
  int window;             // > 0 (with causal): a query at position i sees keys (i - window, i]
  // forms with a sink only
  int keep;               // with a window: keys [0, keep) stay visible to every later query
  const void* temp;       // [nq] per-head factor on the scaled score, or null
  const void* sink;       // [nq] per-head sink logit, or null
  const void* gate;       // gate logits, element (t, h) at gate[t * gate_ld + h], or null
  int64_t gate_ld;
  float slope_base;       // < 0: no distance term
  int vshare = 1;         // consecutive key heads that read one value head (V has nkv / vshare heads)
  int gate_mode = 1;      // gate logits: 1 one per head, 2 one per output element (element (t, h, c) at gate[t * gate_ld + h * D + c])
  int chunk = 0;          // > 0 (window 0): a query sees the keys of its own chunk
  float softcap = 0.f;    // > 0: capped scores
  const float* bias = nullptr;   // [nq, bias_ld], the first n_bias columns are used; distances beyond read the last one
  int n_bias = 0, bias_ld = 0;
  int B = 0, pair_heads = 0, n_head_units = 0;   // set by the launch: sequences, tile pairs over heads, work units per row block
  int* status = nullptr;         // set by the launch: rb_attn_status()
};

}  // namespace rb

// The process's status word of the attention kernels, in pinned host memory that every device can write (null if it cannot be had): not 0 once a
// bounded wait has run out (kStatusGaveUp) or a kernel found its shared memory where it cannot work (kStatusUnaligned), until `rb_attn_wait_error` clears it.  The host reads it without a CUDA call (the bindings do before every launch), the
// optimizer's kernels read it in stream order.
extern "C" int* rb_attn_status();

namespace rb {

constexpr int kStatusGaveUp = 1, kStatusUnaligned = 2;

// At the end of a CTA (all threads): if one of its waits ran out, what it had claimed is missing from the outputs.  Tell the host, and let copies land.
RB_DEVICE void report_given_up(volatile uint32_t* dead, int* status) {
  if (*dead) {
    if (threadIdx.x == 0) {
      *reinterpret_cast<volatile int*>(status) = kStatusGaveUp;
      __threadfence_system();
    }
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    __syncthreads();
  }
}

}  // namespace rb

namespace {

using rb::AttnParams;

constexpr int kMaxSmem = 227 * 1024;

// Every wait is bounded: a wait that runs out sets the CTA's `dead` flag (all later waits of the CTA then return at once), and the
// kernel ends normally after a pause that lets its own copies land; `report_given_up` tells the host.
constexpr int kWaitPolls = 1 << 20;

RB_DEVICE void bounded_wait(uint32_t bar, uint32_t parity, volatile uint32_t* dead) {
  for (int i = 0; !ptx::mbar_try_wait(bar, parity); ++i)
    if (i >= kWaitPolls || *dead) { *dead = 1; return; }
}

RB_DEVICE void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
RB_DEVICE uint4 ld_shared_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
template <typename T> RB_DEVICE uint32_t pack2(float lo, float hi);
template <> RB_DEVICE uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
template <> RB_DEVICE uint32_t pack2<__half>(float lo, float hi) {
  __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// Which sequence a row unit belongs to, units of `rows` rows numbered sequence by sequence; run by a whole warp.  The numbers asked for mostly
// grow, so the search goes on from the last block of 32 sequences.
struct UnitSearch {
  int base = 0, s0 = 0;      // units in front of sequence s0
  // true: `tok0`, `L` of the sequence and the unit's number `r` in it; false: beyond the last sequence
  RB_DEVICE bool find(const int* cu, int B, int rows, int unit, int& tok0, int& L, int& r) {
    const int lane = threadIdx.x & 31;
    if (unit < base) { base = 0; s0 = 0; }
    for (; s0 < B; s0 += 32) {
      const int s = s0 + lane, a = s < B ? cu[s] : 0, len = s < B ? max(cu[s + 1] - a, 0) : 0, c = (len + rows - 1) / rows;
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      const unsigned hit = __ballot_sync(0xffffffffu, base + incl > unit);
      if (hit != 0) {
        const int w = __ffs(hit) - 1;
        tok0 = __shfl_sync(0xffffffffu, a, w);
        L = __shfl_sync(0xffffffffu, len, w);
        r = unit - base - __shfl_sync(0xffffffffu, incl - c, w);
        return true;
      }
      base += __shfl_sync(0xffffffffu, incl, 31);
    }
    base = 0;
    s0 = 0;
    return false;
  }
};

RB_DEVICE float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// cap * tanh(s * scale / cap) + add in the log2 domain, tanh(x) = 1 - 2 / (1 + 2^(2 x log2 e)): c = 2 log2 e * scale / cap,
// k = cap log2 e, k_add = k + add.  Absolute error a few ulp of k; saturates to +-k.
RB_DEVICE float soft_cap2(float s, float c, float k, float k_add) {
  return fmaf(-2.f * k, __fdividef(1.f, 1.f + exp2f(fminf(s * c, 80.f))), k_add);
}

// One instruction for two numbers: (x0, x1) <- (x0, x1) * m + a; (x0, x1) <- (x0, x1) * m + (a0, a1); (s0, s1) <- (s0, s1) + (a0, a1);
// (x0, x1) <- (x0, x1) * (m0, m1)
RB_DEVICE void fma_pair(float& x0, float& x1, float m, float a) {
  asm("{\n\t.reg .b64 x, m, a;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 m, {%2, %2};\n\tmov.b64 a, {%3, %3};\n\tfma.rn.f32x2 x, x, m, a;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(x0), "+f"(x1) : "f"(m), "f"(a));
}
RB_DEVICE void add_pair(float& s0, float& s1, float a0, float a1) {
  asm("{\n\t.reg .b64 s, a;\n\tmov.b64 s, {%0, %1};\n\tmov.b64 a, {%2, %3};\n\tadd.rn.f32x2 s, s, a;\n\tmov.b64 {%0, %1}, s;\n\t}"
      : "+f"(s0), "+f"(s1) : "f"(a0), "f"(a1));
}
RB_DEVICE void fma_pair2(float& x0, float& x1, float m, float a0, float a1) {
  asm("{\n\t.reg .b64 x, m, a;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 m, {%2, %2};\n\tmov.b64 a, {%3, %4};\n\tfma.rn.f32x2 x, x, m, a;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(x0), "+f"(x1) : "f"(m), "f"(a0), "f"(a1));
}
RB_DEVICE void mul_pair(float& x0, float& x1, float m0, float m1) {
  asm("{\n\t.reg .b64 x, m;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 m, {%2, %3};\n\tmul.rn.f32x2 x, x, m;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(x0), "+f"(x1) : "f"(m0), "f"(m1));
}

}  // namespace

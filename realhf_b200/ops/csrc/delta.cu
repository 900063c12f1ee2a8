// Gated delta rule (`DeltaRuleConfig`), packed (prefill) and one-token (decode) forms.  Per head, matrix state S [d, dv] in fp32:
//     S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q          (the output is read after the update; g is one number
//                                                                              or one per row of S)
// All arithmetic that enters the recurrence is fp32; exact expf / log1pf (compiled without fast-math).
//
//   delta_prepare    projection output `proj` [T, ld] = [q (G x d) | k (G x d) | v (H x dv) | ..], beta logits [T, H] and decay inputs
//                    [T, N] (views with their own row stride)  ->  u [T, C + H + N] fp32 = [q | k | v | beta | g],  C = 2 G d + H dv;
//                    N = H: one decay per head, N = H d: one per head and state row:
//                    causal depthwise convolution (taps <= 8, weights [C, taps], tap taps - 1 meets the current token, inputs before a
//                    sequence's first token are zero) + SiLU on the first C channels; q, k <- x / sqrt(sum x^2 + unit_eps) per head, q also times
//                    d^-1/2; beta = sigmoid; g = exp(-exp(A_log of the head) softplus(a + dt_bias)).  Packed form: earlier tokens are the
//                    preceding rows (pos[t] tells how many belong to the sequence), and the last taps - 1 raw inputs of every
//                    sequence go to conv_state [n_slots, taps - 1, C] (oldest first).  Step form (pos == null): earlier inputs
//                    come from conv_state[slot], which is shifted by one.
// Kernels on the decode path are launched with programmatic dependent launch (they signal their successors at once and wait for
// their predecessor before the first global access), like the framework's other decode kernels.
//   delta_rule       the recurrence.  A column of S depends only on its own v column, so columns are independent: a thread group of
//                    LPC lanes owns NC columns (16 state rows of each per lane in registers) or one (32 or 64 rows), a CTA all its groups' columns
//                    of one (sequence, head).  q, k, v, beta, g of 8 tokens at a time are staged in shared memory.  Packed form: S starts
//                    at zero and the final S goes to s_state[slot]; step form: S is loaded from and stored to s_state[slot].
//   gated_head_norm  o / sqrt(mean(o^2) + eps) * w * silu(gate) or sigmoid(gate) per (token, head) -> model type.
#include <type_traits>

#include "anytype.cuh"

namespace {

using rb::ld_any;
using rb::st_any;

constexpr int kMaxTaps = 8;

// write strengths and decays of a token: logits of beta at b[t * ldb + h], decay inputs at a[t * lda + i], i < N (N = H or H * d)
struct GateParams {
  const void* b; int64_t ldb;
  const void* a; int64_t lda;
  const void* A_log; const void* dt_bias;    // [H], [N]
  int N;
};

// decay of input i; rate = exp(A_log) of its head
RB_DEVICE float decay_of(const GateParams& gp, int dt, int64_t t, int i, float rate) {
  const float a = ld_any(gp.a, dt, t * gp.lda + i) + ld_any(gp.dt_bias, dt, i);
  const float sp = a > 20.f ? a : log1pf(expf(a));
  return expf(-rate * sp);
}

// Gate units of the prepare kernels (grid.y from 2 G + H on): the first one writes the strengths, and the decays when there is one
// per head; with one decay per state row, H further units follow, one per head.
RB_DEVICE void gate_unit(const GateParams& gp, float* u, int dt, int unit, int64_t t0, int nt, int H, int C, int UW) {
  const int per = gp.N / H;
  if (unit == 0) {
    for (int idx = threadIdx.x; idx < nt * H; idx += blockDim.x) {
      const int64_t t = t0 + idx / H;
      const int h = idx % H;
      u[t * UW + C + h] = 1.f / (1.f + expf(-ld_any(gp.b, dt, t * gp.ldb + h)));
      if (per == 1) u[t * UW + C + H + h] = decay_of(gp, dt, t, h, expf(ld_any(gp.A_log, dt, h)));
    }
    return;
  }
  const int h = unit - 1;
  const float rate = expf(ld_any(gp.A_log, dt, h));
  for (int idx = threadIdx.x; idx < nt * per; idx += blockDim.x) {
    const int64_t t = t0 + idx / per;
    const int i = h * per + idx % per;
    u[t * UW + C + H + i] = decay_of(gp, dt, t, i, rate);
  }
}

// One CTA per (token, unit); a unit is a q or k head, a v head, or a gate unit (as in the tiled kernel below), so that a decode batch
// of a few rows still spreads over the GPU.
__global__ void __launch_bounds__(128) delta_prepare_kernel(const void* __restrict__ proj, int64_t ld, int dt, const void* __restrict__ conv_w,
                                                            GateParams gp, float* __restrict__ u, const int* __restrict__ pos,
                                                            float* __restrict__ conv_state,
                                                            const int* __restrict__ tok_slot, const int* __restrict__ remain,
                                                            const int* __restrict__ slots, int H, int G, int d, int dv, int taps,
                                                            float unit_eps) {
  extern __shared__ float ys[];               // [channels of the unit] convolved + SiLU
  __shared__ float red[32];
  const int64_t t = blockIdx.x;
  const int unit = blockIdx.y;
  const int nqk = G * d, nv = H * dv, C = 2 * nqk + nv, UW = C + H + gp.N;
  rb::pdl_trigger();
  rb::pdl_wait();
  if (unit >= 2 * G + H) {
    gate_unit(gp, u, dt, unit - 2 * G - H, t, 1, H, C, UW);
    return;
  }
  const bool is_qk = unit < 2 * G;
  const int us = is_qk ? d : dv;
  const int c_base = is_qk ? unit * d : 2 * nqk + (unit - 2 * G) * dv;
  const bool step = pos == nullptr;
  const int p = step ? 0 : pos[t];
  int slot = -1;
  if (conv_state != nullptr) slot = step ? (slots ? slots[t] : (int)t) : tok_slot[t];
  const int rem = (!step && conv_state != nullptr) ? remain[t] : 0;
  float* st = (slot >= 0 && taps > 1) ? conv_state + (int64_t)slot * (taps - 1) * C : nullptr;
  float ss = 0.f;
  for (int cl = threadIdx.x; cl < us; cl += blockDim.x) {
    const int c = c_base + cl;
    const float x = ld_any(proj, dt, t * ld + c);
    float hist[kMaxTaps - 1];
    float y = 0.f;
#pragma unroll
    for (int back = kMaxTaps - 1; back >= 1; --back) {       // oldest first, the current token last: the tiled kernel's order
      if (back < taps) {
        float xb;
        if (step) xb = st ? st[(int64_t)(taps - 1 - back) * C + c] : 0.f;
        else xb = back <= p ? ld_any(proj, dt, (t - back) * ld + c) : 0.f;
        hist[back - 1] = xb;
        y = fmaf(xb, ld_any(conv_w, dt, (int64_t)c * taps + taps - 1 - back), y);
      }
    }
    y = fmaf(x, ld_any(conv_w, dt, (int64_t)c * taps + taps - 1), y);
    if (st != nullptr) {
      if (step) {           // shift: row i <- row i + 1, the newest row <- x (this thread owns channel c of the slot)
#pragma unroll
        for (int back = kMaxTaps - 1; back >= 1; --back)
          if (back < taps) st[(int64_t)(taps - 1 - back) * C + c] = back == 1 ? x : hist[back - 2];
      } else if (rem < taps - 1) {
        st[(int64_t)(taps - 2 - rem) * C + c] = x;
      }
    }
    y = y / (1.f + expf(-y));
    ys[cl] = y;
    ss = fmaf(y, y, ss);
  }
  float r = 1.f;
  if (is_qk) {
    ss = rb::block_reduce<false>(ss, red);
    r = 1.f / sqrtf(ss + unit_eps);
    if (unit < G) r *= 1.f / sqrtf((float)d);
  }
  for (int cl = threadIdx.x; cl < us; cl += blockDim.x) u[t * UW + c_base + cl] = ys[cl] * r;   // a thread re-reads its own entries
}

// Packed form for long batches: a CTA owns 16 consecutive tokens x one unit of channels (a q or k head, a v head, or a gate unit).
// A thread keeps its channels' taps and a sliding window of the last taps - 1 inputs in registers and walks the tokens,
// so every input is read once (plus a halo of taps - 1 rows per tile) and the weights once per CTA; the per-(token, head) sums of
// squares are reduced per warp into shared memory and applied after one barrier.
constexpr int kPT = 16, kPThreads = 128;   // tokens per tile, threads; CH channels per thread (units of up to CH * 128 channels)

template <int CH>
__global__ void __launch_bounds__(kPThreads) delta_prepare_tiled_kernel(const void* __restrict__ proj, int64_t ld, int dt, const void* __restrict__ conv_w,
                                                                        GateParams gp, float* __restrict__ u, const int* __restrict__ pos,
                                                                        float* __restrict__ conv_state, const int* __restrict__ tok_slot,
                                                                        const int* __restrict__ remain, int64_t T, int H, int G, int d, int dv,
                                                                        int taps, float unit_eps) {
  __shared__ float part[kPThreads / 32][kPT];
  const int nqk = G * d, nv = H * dv, C = 2 * nqk + nv, UW = C + H + gp.N;
  const int unit = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t t0 = (int64_t)blockIdx.x * kPT;
  const int nt = (int)min((int64_t)kPT, T - t0);
  if (unit >= 2 * G + H) {
    gate_unit(gp, u, dt, unit - 2 * G - H, t0, nt, H, C, UW);
    return;
  }
  const bool is_qk = unit < 2 * G;
  const int us = is_qk ? d : dv;                       // channels of this unit
  const int c_base = is_qk ? unit * d : 2 * nqk + (unit - 2 * G) * dv;
  // all loads of the tile first (independent, in flight together), then the arithmetic
  int ps[kPT];
#pragma unroll
  for (int tt = 0; tt < kPT; ++tt) ps[tt] = tt < nt ? pos[t0 + tt] : 0;
  float w[CH][kMaxTaps], hist[CH][kMaxTaps - 1], xv[CH][kPT];
  bool okc[CH];
#pragma unroll
  for (int ch = 0; ch < CH; ++ch) {
    okc[ch] = tid + ch * kPThreads < us;
    const int c = c_base + tid + ch * kPThreads;
#pragma unroll
    for (int tt = 0; tt < kPT; ++tt) xv[ch][tt] = (okc[ch] && tt < nt) ? ld_any(proj, dt, (t0 + tt) * ld + c) : 0.f;
#pragma unroll
    for (int back = 0; back < kMaxTaps; ++back)      // w[ch][back]: the tap that meets the input `back` tokens ago
      w[ch][back] = (okc[ch] && back < taps) ? ld_any(conv_w, dt, (int64_t)c * taps + taps - 1 - back) : 0.f;
#pragma unroll
    for (int back = 1; back < kMaxTaps; ++back)
      hist[ch][back - 1] = (okc[ch] && back < taps && t0 - back >= 0) ? ld_any(proj, dt, (t0 - back) * ld + c) : 0.f;
  }
  if (conv_state != nullptr && taps > 1) {
#pragma unroll
    for (int tt = 0; tt < kPT; ++tt) {
      if (tt < nt) {
        const int slot = tok_slot[t0 + tt], rem = remain[t0 + tt];
        if (slot >= 0 && rem < taps - 1) {
#pragma unroll
          for (int ch = 0; ch < CH; ++ch)
            if (okc[ch]) conv_state[((int64_t)slot * (taps - 1) + (taps - 2 - rem)) * C + c_base + tid + ch * kPThreads] = xv[ch][tt];
        }
      }
    }
  }
#pragma unroll
  for (int tt = 0; tt < kPT; ++tt) {
    float ss = 0.f;
    if (tt < nt) {
      const int p = ps[tt];
#pragma unroll
      for (int ch = 0; ch < CH; ++ch) {
        const float x = xv[ch][tt];
        float y = 0.f;
#pragma unroll
        for (int back = kMaxTaps - 1; back >= 1; --back)      // oldest first, the current token last: a fixed order
          if (back < taps && back <= p) y = fmaf(hist[ch][back - 1], w[ch][back], y);
        y = fmaf(x, w[ch][0], y);
#pragma unroll
        for (int back = kMaxTaps - 1; back >= 2; --back) hist[ch][back - 1] = hist[ch][back - 2];
        hist[ch][0] = x;
        y = y / (1.f + expf(-y));
        xv[ch][tt] = y;
        ss = fmaf(y, y, ss);
      }
    }
    if (is_qk) {
      ss = rb::warp_sum(ss);
      if (lane == 0) part[warp][tt] = ss;
    }
  }
  if (is_qk) __syncthreads();
#pragma unroll
  for (int tt = 0; tt < kPT; ++tt) {
    if (tt < nt) {
      float r = 1.f;
      if (is_qk) {
        r = 1.f / sqrtf(part[0][tt] + part[1][tt] + part[2][tt] + part[3][tt] + unit_eps);
        if (unit < G) r *= 1.f / sqrtf((float)d);
      }
#pragma unroll
      for (int ch = 0; ch < CH; ++ch)
        if (okc[ch]) u[(t0 + tt) * UW + c_base + tid + ch * kPThreads] = xv[ch][tt] * r;
    }
  }
}

// The same for head sizes in whole fours up to 128 on aligned rows: a warp owns one unit of channels, four neighbouring ones a lane, and walks kWalk
// tokens in tiles of 8 whose rows it has in flight together; the per-(token, head) sum of squares stays inside the warp.  The kernel above moves two
// bytes a lane and load and four a store, and waits for its loads with few of them on their way: 8 sequences of 700 .. 1024 tokens, 16 + 2 x 4 heads x 128
// (71 MB in, 85 MB out) 121 us; this way 49.  What it waits for is its loads and the issue of some 45 instructions a channel and token (24 us of bytes, about 20
// of issue), so rows on their way stay as they are in memory: 94 registers and five CTAs an SM for 16-bit rows (widened on arrival, the type told apart at
// run time, 124 registers: 87 us; four CTAs 57, six, with spills, 53; bf16 widened by the pair conversions instead of shifts 59).  kTaps: the taps that registers are kept for.
constexpr int kTile = 8;

template <typename T4, int kTaps, int kWalk>
__global__ void __launch_bounds__(kPThreads, kTaps > 4 ? 3 : (sizeof(T4) == 2 ? 5 : 4)) delta_prepare_warp_kernel(const void* __restrict__ proj, int64_t ld, int dt, const void* __restrict__ conv_w,
                                                                       GateParams gp, float* __restrict__ u, const int* __restrict__ pos,
                                                                       float* __restrict__ conv_state, const int* __restrict__ tok_slot,
                                                                       const int* __restrict__ remain, int64_t T, int H, int G, int d, int dv,
                                                                       int taps, float unit_eps) {
  const int nqk = G * d, nv = H * dv, C = 2 * nqk + nv, UW = C + H + gp.N;
  const int unit = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kPerCta = kPThreads / 32 * kWalk;
  const int64_t b0 = (int64_t)blockIdx.y * kPerCta;
  if (unit >= 2 * G + H) {
    gate_unit(gp, u, dt, unit - 2 * G - H, b0, (int)min((int64_t)kPerCta, T - b0), H, C, UW);
    return;
  }
  const int64_t t0 = b0 + warp * kWalk;
  const int nt = (int)min((int64_t)kWalk, T - t0);
  if (nt <= 0) return;
  const bool is_qk = unit < 2 * G, mine = lane * 4 < (is_qk ? d : dv);
  const int c = (is_qk ? unit * d : 2 * nqk + (unit - 2 * G) * dv) + lane * 4;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  using Raw = std::conditional_t<sizeof(T4) == 2, uint2, float4>;   // rows on their way stay as they are in memory
  const T4* rows = static_cast<const T4*>(proj) + t0 * ld + c;
  auto load = [&](int i) { return mine && i < nt ? *reinterpret_cast<const Raw*>(rows + i * ld) : Raw{}; };
  auto wide = [](const Raw& r) {
    if constexpr (std::is_same_v<T4, __nv_bfloat16>)
      return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xffff0000u));
    else
      return rb::ld4_any(&r, sizeof(T4) == 4 ? 0 : 2, 0);
  };
  float4 w[kTaps], hist[kTaps - 1];                       // w[back]: the taps that meet the input `back` tokens ago; hist[back - 1]: that input
  Raw xr[kTile];
#pragma unroll
  for (int i = 0; i < kTile; ++i) xr[i] = load(i);
#pragma unroll
  for (int back = 1; back < kTaps; ++back) hist[back - 1] = mine && back < taps && t0 - back >= 0 ? wide(*reinterpret_cast<const Raw*>(rows - back * ld)) : zero;
#pragma unroll
  for (int back = 0; back < kTaps; ++back) {
    const bool in = mine && back < taps;
    const int64_t at = (int64_t)c * taps + taps - 1 - back;
    w[back] = in ? make_float4(ld_any(conv_w, dt, at), ld_any(conv_w, dt, at + taps), ld_any(conv_w, dt, at + 2 * taps), ld_any(conv_w, dt, at + 3 * taps)) : zero;
  }
  const float scale = unit < G ? 1.f / sqrtf((float)d) : 1.f;
  for (int s0 = 0; s0 < nt; s0 += kTile) {
    const int p0 = lane < kTile && s0 + lane < nt ? pos[t0 + s0 + lane] : 0;
    Raw nx[kTile];                                        // the next tile's rows
#pragma unroll
    for (int i = 0; i < kTile; ++i) nx[i] = load(s0 + kTile + i);
    if (conv_state != nullptr && taps > 1) {
#pragma unroll
      for (int i = 0; i < kTile; ++i)
        if (s0 + i < nt) {
          const int slot = tok_slot[t0 + s0 + i], rem = remain[t0 + s0 + i];
          if (slot >= 0 && rem < taps - 1 && mine) {
            float* st = conv_state + ((int64_t)slot * (taps - 1) + (taps - 2 - rem)) * C + c;
            const float4 x = wide(xr[i]);
            st[0] = x.x; st[1] = x.y; st[2] = x.z; st[3] = x.w;
          }
        }
    }
#pragma unroll
    for (int i = 0; i < kTile; ++i) {
      const int p = __shfl_sync(0xffffffffu, p0, i);
      float4 y = zero;
      const float4 x = wide(xr[i]);
      auto tap = [&](const float4& a, const float4& b) {
        y.x = fmaf(a.x, b.x, y.x); y.y = fmaf(a.y, b.y, y.y); y.z = fmaf(a.z, b.z, y.z); y.w = fmaf(a.w, b.w, y.w);
      };
#pragma unroll
      for (int back = kTaps - 1; back >= 1; --back)       // oldest first, the current token last: a fixed order
        if (back < taps && back <= p) tap(hist[back - 1], w[back]);
      tap(x, w[0]);
#pragma unroll
      for (int back = kTaps - 1; back >= 2; --back) hist[back - 1] = hist[back - 2];
      if constexpr (kTaps > 1) hist[0] = x;
      y.x = y.x / (1.f + expf(-y.x)); y.y = y.y / (1.f + expf(-y.y)); y.z = y.z / (1.f + expf(-y.z)); y.w = y.w / (1.f + expf(-y.w));
      if (is_qk) {
        const float r = scale * (1.f / sqrtf(rb::warp_sum((y.x * y.x + y.y * y.y) + (y.z * y.z + y.w * y.w)) + unit_eps));
        y.x *= r; y.y *= r; y.z *= r; y.w *= r;
      }
      if (mine && s0 + i < nt) *reinterpret_cast<float4*>(u + (t0 + s0 + i) * UW + c) = y;
    }
#pragma unroll
    for (int i = 0; i < kTile; ++i) xr[i] = nx[i];
  }
}

// ------------------------------------------------------------------------------------------------ recurrence
constexpr int kScanThreads = 128, kTok = 8;

struct ScanParams {
  const float* u; float* o;
  const int* cu;            // packed form: [n_seqs + 1]; step form: null (sequence b = row b, one token)
  float* s_state;           // [n_slots, H, d, dv] or null
  const int* slots;         // per sequence / row; null = identity (step form) or no state (packed form)
  int H, G, d, dv, step;
  int vec = 0;              // rows of s_state may be written 16 bytes at a time
};

// Packed form.  A group of LPC lanes owns NC neighbouring columns of the state: lane l holds their rows ((e / 4) * LPC + l) * 4 + e % 4, e = 0 .. 15, so that its q / k
// operands are four aligned float4 reads of shared memory each per token, used for all NC columns.  kChan: a decay per state row, staged beside q and k.
//
// What bounds it: a token is one step of a serial chain, so what counts is its latency and, with few sequences, the shared-memory port and the fp32
// pipe of the SMs that hold two CTAs.  With D the decayed state, the output is S^T q = D^T q + (k . q) u: both products read D, none waits for the
// update, and k . q is one number per token for all columns.  A scalar decay is not multiplied into the state: S = c Z with c the product of the
// decays since the last time Z took it in, u enters Z as u / c, and Z takes c in when c falls below 2^-20 (at once for a decay of 0).  That leaves three
// multiply-adds per state element and token, two elements an instruction.  8 sequences of 700..1024 tokens, 16 heads x 128 x 128: 643 us with the
// decay, the update and the second product in sequence and one column per lane pair; 595 us with this order (a lane of a column's pair reads 32
// float4s of q and k a token, and shared memory serves an SM one such read in four cycles); 540 us with four columns to a group of eight lanes.
RB_DEVICE uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
RB_DEVICE uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
RB_DEVICE uint64_t pair_of(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
RB_DEVICE float2 halves(uint64_t a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
constexpr float kTakeIn = 1.f / (1 << 20);

template <int LPC, int NC, bool kChan>
__global__ void __launch_bounds__(kScanThreads, LPC <= 8 ? 3 : 2) delta_rule_kernel(ScanParams p) {
  constexpr int kRows = 16, NCOL = kScanThreads / LPC * NC;
  static_assert(2 * NC <= LPC, "a lane ends up with at most one of the group's 2 NC sums");
  extern __shared__ __align__(16) float sm[];
  __shared__ float4 tok[kTok];                     // per token: beta, c after its decay, 1 / c (0: Z takes c in), k . q
  const int seq = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * NCOL;
  const int g = h / (p.H / p.G), d = p.d, dv = p.dv;
  const int nqk = p.G * d, C = 2 * nqk + p.H * dv, UW = C + p.H + (kChan ? p.H * d : p.H);
  const int tid = threadIdx.x, l = tid % LPC, lcol = tid / LPC * NC, col = c0 + lcol, warp = tid >> 5, lane = tid & 31;
  rb::pdl_trigger();
  rb::pdl_wait();
  const int t0 = p.cu[seq], t1 = p.cu[seq + 1];
  if (t1 <= t0) return;
  const int slot = p.s_state == nullptr || p.slots == nullptr ? -1 : p.slots[seq];
  float* S_g = slot >= 0 ? p.s_state + (((int64_t)slot * p.H + h) * d) * dv : nullptr;
  constexpr int dpad = kRows * LPC;               // rows >= d hold zeros and read zero q / k
  constexpr int kBuf = (kChan ? 3 : 2) * kTok * dpad + kTok * NCOL + 2 * kTok;   // floats of one staging buffer: q, k, v, (beta, g), row decays
  constexpr int NQ = kTok * dpad / kScanThreads, NV = (kTok * NCOL + kScanThreads - 1) / kScanThreads;
  auto row_of = [&](int e) { return ((e >> 2) * LPC + l) * 4 + (e & 3); };
  // Up to 16 lanes the zeros start at an index that the compiler cannot know to be 0 (no head count is negative), so they reach the registers through local
  // memory, once: with constants in front of it the token loop gets a worse schedule (8 sequences of 700..1024 tokens, 16 heads x 128 x 128: 687 us
  // against 620, the whole prefill 715 against 669; with registers for four CTAs an SM 612 and 703).  For 32 lanes constants are better (2 x 512 tokens,
  // 4 heads x 512 x 512: 372 us against 395).
  const int first = LPC < 32 ? min(p.H, 0) : 0;
  uint64_t Z[NC][kRows / 2];
#pragma unroll
  for (int j = 0; j < NC; ++j)
#pragma unroll
    for (int e = first; e < kRows / 2; ++e) Z[j][e] = 0;
  // The inputs of the next 8 tokens are fetched into registers while the current 8 are processed out of shared memory (two staging buffers).
  float rq[NQ], rk[NQ], rg[kChan ? NQ : 1], rv[NV], rb = 0.f;
  auto fetch = [&](int tb) {
    const int nt = min(kTok, t1 - tb);
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
      const int idx = tid + i * kScanThreads, tt = idx / dpad, e = idx % dpad;
      const bool ok = tt < nt && e < d;
      const float* row = p.u + (int64_t)(tb + tt) * UW;
      rq[i] = ok ? row[g * d + e] : 0.f;
      rk[i] = ok ? row[nqk + g * d + e] : 0.f;
      if constexpr (kChan) rg[i] = ok ? row[C + p.H + h * d + e] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int idx = tid + i * kScanThreads, tt = idx / NCOL, c = c0 + idx % NCOL;
      rv[i] = (idx < kTok * NCOL && tt < nt && c < dv) ? p.u[(int64_t)(tb + tt) * UW + 2 * nqk + h * dv + c] : 0.f;
    }
    rb = (tid < nt * 2 && !(kChan && (tid & 1))) ? p.u[(int64_t)(tb + tid / 2) * UW + C + (tid & 1) * p.H + h] : 0.f;
  };
  auto stage = [&](float* buf) {
#pragma unroll
    for (int i = 0; i < NQ; ++i) { buf[tid + i * kScanThreads] = rq[i]; buf[kTok * dpad + tid + i * kScanThreads] = rk[i]; }
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (tid + i * kScanThreads < kTok * NCOL) buf[2 * kTok * dpad + tid + i * kScanThreads] = rv[i];
    if (tid < 2 * kTok) buf[2 * kTok * dpad + kTok * NCOL + tid] = rb;
    if constexpr (kChan) {
#pragma unroll
      for (int i = 0; i < NQ; ++i) buf[2 * kTok * dpad + kTok * NCOL + 2 * kTok + tid + i * kScanThreads] = rg[i];
    }
  };
  // which of the group's sums (k products of its NC columns, then q products) this lane ends up with
  int mine = 0;
#pragma unroll
  for (int n = 2 * NC, o = LPC / 2; n > 1; n >>= 1, o >>= 1) mine += (l & o) ? n / 2 : 0;
  const int my_col = mine % NC;
  const bool writes = mine >= NC && (l & (LPC / (2 * NC) - 1)) == 0 && col + my_col < dv;

  fetch(t0);
  int which = 0;
  float c = 1.f;                                   // S = c Z (the same in all threads)
  for (int tb = t0; tb < t1; tb += kTok, which ^= 1) {
    const int nt = min(kTok, t1 - tb);
    float* buf = sm + which * kBuf;
    stage(buf);
    __syncthreads();                               // (the numbers of the last chunk's tokens have been read, too)
    const float* qs = buf;
    const float* ks = buf + kTok * dpad;
    const float* vs = ks + kTok * dpad;
    const float* bg = vs + kTok * NCOL;
    const float* gs = bg + 2 * kTok;                // kChan: [kTok][dpad]
    // the chunk's numbers per token: every warp k . q of two tokens, the decays' products in every lane, one token's kept
    float c1 = 1.f, beta1 = 0.f;
    bool in1 = false;
#pragma unroll
    for (int tt = 0; tt < kTok; ++tt) {
      if constexpr (!kChan) c *= tt < nt ? bg[tt * 2 + 1] : 1.f;
      const bool in = !kChan && !(c >= kTakeIn && c <= 1.f / kTakeIn);
      if (lane == tt) { c1 = c; in1 = in; beta1 = bg[tt * 2]; }
      if (in) c = 1.f;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int tt = warp + 4 * i;
      float a = 0.f;
#pragma unroll
      for (int e = 0; e < dpad; e += 32) a = fmaf(ks[tt * dpad + e + lane], qs[tt * dpad + e + lane], a);
      a = rb::warp_sum(a);
      if (lane == tt) tok[tt] = make_float4(beta1, c1, in1 ? 0.f : 1.f / c1, a);
    }
    __syncthreads();
    if (tb + kTok < t1) fetch(tb + kTok);
    for (int tt = 0; tt < nt; ++tt) {
      const float4 n = tok[tt];
      const ulonglong2* kp = reinterpret_cast<const ulonglong2*>(ks + tt * dpad) + l;
      const ulonglong2* qp = reinterpret_cast<const ulonglong2*>(qs + tt * dpad) + l;
      const float v = vs[tt * NCOL + lcol + my_col];
      uint64_t kk[kRows / 2], ak[NC], aq[NC];
#pragma unroll
      for (int j = 0; j < NC; ++j) ak[j] = aq[j] = 0;
#pragma unroll
      for (int e4 = 0; e4 < kRows / 4; ++e4) {
        const ulonglong2 k2 = kp[e4 * LPC], q2 = qp[e4 * LPC];
        kk[2 * e4] = k2.x;
        kk[2 * e4 + 1] = k2.y;
        if constexpr (kChan) {
          const ulonglong2 g2 = (reinterpret_cast<const ulonglong2*>(gs + tt * dpad) + l)[e4 * LPC];
#pragma unroll
          for (int j = 0; j < NC; ++j) {
            Z[j][2 * e4] = mul2(Z[j][2 * e4], g2.x);
            Z[j][2 * e4 + 1] = mul2(Z[j][2 * e4 + 1], g2.y);
          }
        }
#pragma unroll
        for (int j = 0; j < NC; ++j) { ak[j] = fma2(Z[j][2 * e4], k2.x, ak[j]); aq[j] = fma2(Z[j][2 * e4], q2.x, aq[j]); }
#pragma unroll
        for (int j = 0; j < NC; ++j) { ak[j] = fma2(Z[j][2 * e4 + 1], k2.y, ak[j]); aq[j] = fma2(Z[j][2 * e4 + 1], q2.y, aq[j]); }
      }
      float sum[2 * NC];
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        const float2 a = halves(ak[j]), b = halves(aq[j]);
        sum[j] = a.x + a.y;
        sum[NC + j] = b.x + b.y;
      }
      // the group's sums over its lanes: every step halves what a lane still carries, then the rest is summed whole
#pragma unroll
      for (int m = 2 * NC, o = LPC / 2; m > 1; m >>= 1, o >>= 1) {
        const bool hi = (l & o) != 0;
#pragma unroll
        for (int i = 0; i < m / 2; ++i) {
          const float keep = hi ? sum[m / 2 + i] : sum[i], send = hi ? sum[i] : sum[m / 2 + i];
          sum[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
#pragma unroll
      for (int o = LPC / (2 * NC) / 2; o > 0; o >>= 1) sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], o);
      const float w = n.x * (v - n.y * sum[0]);                                      // (meaningful in the lanes that hold a k product)
      const float w_mine = __shfl_xor_sync(0xffffffffu, w, LPC / 2);                 // the same column's, in the lanes that hold a q product
      if (writes) p.o[((int64_t)(tb + tt) * p.H + h) * dv + col + my_col] = fmaf(w_mine, n.w, n.y * sum[0]);
      const bool take = !kChan && n.z == 0.f;
      const uint64_t c2 = pair_of(n.y, n.y);
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        float wj = __shfl_sync(0xffffffffu, w, (lane & ~(LPC - 1)) + j * (LPC / (2 * NC)));     // lane that holds sum j
        if (take) {
#pragma unroll
          for (int e = 0; e < kRows / 2; ++e) Z[j][e] = mul2(Z[j][e], c2);
        } else {
          wj *= n.z;
        }
        const uint64_t w2 = pair_of(wj, wj);
#pragma unroll
        for (int e = 0; e < kRows / 2; ++e) Z[j][e] = fma2(kk[e], w2, Z[j][e]);
      }
    }
  }
  if (S_g && NC == 4 && p.vec) {
    if (col < dv) {
#pragma unroll
      for (int e = 0; e < kRows; ++e) {
        float z[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) { const float2 v = halves(Z[j % NC][e / 2]); z[j] = c * (e & 1 ? v.y : v.x); }
        if (row_of(e) < d) *reinterpret_cast<float4*>(S_g + (int64_t)row_of(e) * dv + col) = make_float4(z[0], z[1], z[2], z[3]);
      }
    }
  } else if (S_g) {
#pragma unroll
    for (int j = 0; j < NC; ++j)
#pragma unroll
      for (int e = 0; e < kRows; e += 2) {
        const float2 z = halves(Z[j][e / 2]);
        if (col + j < dv && row_of(e) < d) S_g[(int64_t)row_of(e) * dv + col + j] = c * z.x;
        if (col + j < dv && row_of(e + 1) < d) S_g[(int64_t)row_of(e + 1) * dv + col + j] = c * z.y;
      }
  }
}

// Step form: one token per row, and reading and writing the state is all the work.  A thread group of LPC lanes owns one column (32 or 64 state rows
// per lane), so that every access of a warp to the state covers whole 32-byte sectors.  The packed form of head sizes up to 64 also runs here, where
// sharing q and k between columns saves little: size 64, 8 heads, 2 x 512 / 64 x 100 tokens 142 / 77 us against 166 / 84; size 32 110 / 59 against 122 / 43,
// so many CTAs of size 32 take the other kernel.  (With the packed form's eight lanes and four columns an access
// touched 16 sectors for a quarter each: 16 heads x 128 x 128, 1 / 16 / 128 rows 6.1 / 17.9 / 110 us, against 3.8 / 8.9 / 67.6 this way.)
// Row mapping: lane l of a column's LPC lanes holds the state rows ((e / 4) * LPC + l) * 4 + e % 4, e = 0 .. kEPL - 1, so that its q / k
// operands are 8 aligned float4 reads of shared memory per token (the lanes of a column read neighbouring float4s, the columns of
// a warp the same ones).  Dot products run on four independent accumulators.  kChan: a decay per state row, staged beside q and k.
template <int LPC, int kEPL, bool kChan>
__global__ void __launch_bounds__(kScanThreads, kEPL == 32 ? 3 : 2) delta_column_kernel(ScanParams p) {
  constexpr int NCOL = kScanThreads / LPC;
  extern __shared__ __align__(16) float sm[];
  const int seq = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * NCOL;
  const int g = h / (p.H / p.G), d = p.d, dv = p.dv;
  const int nqk = p.G * d, C = 2 * nqk + p.H * dv, UW = C + p.H + (kChan ? p.H * d : p.H);
  const int tid = threadIdx.x, l = tid % LPC, col = c0 + tid / LPC;
  const bool active = col < dv;
  int t0, t1;
  rb::pdl_trigger();
  rb::pdl_wait();
  if (p.step) { t0 = seq; t1 = seq + 1; } else { t0 = p.cu[seq]; t1 = p.cu[seq + 1]; }
  if (t1 <= t0) return;
  const int slot = p.s_state == nullptr ? -1 : (p.slots ? p.slots[seq] : (p.step ? seq : -1));
  float* S_g = slot >= 0 ? p.s_state + (((int64_t)slot * p.H + h) * d) * dv : nullptr;
  constexpr int dpad = kEPL * LPC;                // rows >= d hold zeros and read zero q / k
  constexpr int kBuf = (kChan ? 3 : 2) * kTok * dpad + kTok * NCOL + 2 * kTok;   // floats of one staging buffer: q, k, v, (beta, g), row decays
  constexpr int NQ = kTok * dpad / kScanThreads, NV = (kTok * NCOL + kScanThreads - 1) / kScanThreads;
  auto row_of = [&](int e) { return ((e >> 2) * LPC + l) * 4 + (e & 3); };
  float S[kEPL];
#pragma unroll
  for (int e = 0; e < kEPL; ++e) {
    const int row = row_of(e);
    S[e] = (p.step && S_g && active && row < d) ? S_g[(int64_t)row * dv + col] : 0.f;
  }
  // The inputs of the next 8 tokens are fetched into registers while the current 8 are processed out of shared memory (two
  // staging buffers, one barrier per chunk).
  float rq[NQ], rk[NQ], rg[kChan ? NQ : 1], rv[NV], rb = 0.f;
  auto fetch = [&](int tb) {
    const int nt = min(kTok, t1 - tb);
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
      const int idx = tid + i * kScanThreads, tt = idx / dpad, e = idx % dpad;
      const bool ok = tt < nt && e < d;
      const float* row = p.u + (int64_t)(tb + tt) * UW;
      rq[i] = ok ? row[g * d + e] : 0.f;
      rk[i] = ok ? row[nqk + g * d + e] : 0.f;
      if constexpr (kChan) rg[i] = ok ? row[C + p.H + h * d + e] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int idx = tid + i * kScanThreads, tt = idx / NCOL, c = c0 + idx % NCOL;
      rv[i] = (idx < kTok * NCOL && tt < nt && c < dv) ? p.u[(int64_t)(tb + tt) * UW + 2 * nqk + h * dv + c] : 0.f;
    }
    rb = (tid < nt * 2 && !(kChan && (tid & 1))) ? p.u[(int64_t)(tb + tid / 2) * UW + C + (tid & 1) * p.H + h] : 0.f;
  };
  auto stage = [&](float* buf) {
#pragma unroll
    for (int i = 0; i < NQ; ++i) { buf[tid + i * kScanThreads] = rq[i]; buf[kTok * dpad + tid + i * kScanThreads] = rk[i]; }
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (tid + i * kScanThreads < kTok * NCOL) buf[2 * kTok * dpad + tid + i * kScanThreads] = rv[i];
    if (tid < 2 * kTok) buf[2 * kTok * dpad + kTok * NCOL + tid] = rb;
    if constexpr (kChan) {
#pragma unroll
      for (int i = 0; i < NQ; ++i) buf[2 * kTok * dpad + kTok * NCOL + 2 * kTok + tid + i * kScanThreads] = rg[i];
    }
  };
  fetch(t0);
  int which = 0;
  for (int tb = t0; tb < t1; tb += kTok, which ^= 1) {
    const int nt = min(kTok, t1 - tb);
    float* buf = sm + which * kBuf;
    stage(buf);
    __syncthreads();
    if (tb + kTok < t1) fetch(tb + kTok);
    const float* qs = buf;
    const float* ks = buf + kTok * dpad;
    const float* vs = ks + kTok * dpad;
    const float* bg = vs + kTok * NCOL;
    const float* gs = bg + 2 * kTok;                // kChan: [kTok][dpad]
    for (int tt = 0; tt < nt; ++tt) {
      const float beta = bg[tt * 2], gg = bg[tt * 2 + 1];
      const float4* kq = reinterpret_cast<const float4*>(ks + tt * dpad) + l;
      const float4* qq = reinterpret_cast<const float4*>(qs + tt * dpad) + l;
      const float4* dg = reinterpret_cast<const float4*>(gs + tt * dpad) + l;
      float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
      for (int e4 = 0; e4 < kEPL / 4; ++e4) {
        const float4 kk = kq[e4 * LPC];
        if constexpr (kChan) {
          const float4 g4 = dg[e4 * LPC];
          S[e4 * 4] *= g4.x; S[e4 * 4 + 1] *= g4.y; S[e4 * 4 + 2] *= g4.z; S[e4 * 4 + 3] *= g4.w;
        } else {
          S[e4 * 4] *= gg; S[e4 * 4 + 1] *= gg; S[e4 * 4 + 2] *= gg; S[e4 * 4 + 3] *= gg;
        }
        a0 = fmaf(S[e4 * 4], kk.x, a0); a1 = fmaf(S[e4 * 4 + 1], kk.y, a1);
        a2 = fmaf(S[e4 * 4 + 2], kk.z, a2); a3 = fmaf(S[e4 * 4 + 3], kk.w, a3);
      }
      float acc = (a0 + a1) + (a2 + a3);
#pragma unroll
      for (int off = 1; off < LPC; off <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
      const float w = beta * (vs[tt * NCOL + tid / LPC] - acc);
      a0 = a1 = a2 = a3 = 0.f;
#pragma unroll
      for (int e4 = 0; e4 < kEPL / 4; ++e4) {
        const float4 kk = kq[e4 * LPC], q4 = qq[e4 * LPC];
        S[e4 * 4] = fmaf(kk.x, w, S[e4 * 4]); S[e4 * 4 + 1] = fmaf(kk.y, w, S[e4 * 4 + 1]);
        S[e4 * 4 + 2] = fmaf(kk.z, w, S[e4 * 4 + 2]); S[e4 * 4 + 3] = fmaf(kk.w, w, S[e4 * 4 + 3]);
        a0 = fmaf(S[e4 * 4], q4.x, a0); a1 = fmaf(S[e4 * 4 + 1], q4.y, a1);
        a2 = fmaf(S[e4 * 4 + 2], q4.z, a2); a3 = fmaf(S[e4 * 4 + 3], q4.w, a3);
      }
      float ov = (a0 + a1) + (a2 + a3);
#pragma unroll
      for (int off = 1; off < LPC; off <<= 1) ov += __shfl_xor_sync(0xffffffffu, ov, off);
      if (active && l == 0) p.o[((int64_t)(tb + tt) * p.H + h) * dv + col] = ov;
    }
  }
  if (S_g && active) {
#pragma unroll
    for (int e = 0; e < kEPL; ++e) {
      const int row = row_of(e);
      if (row < d) S_g[(int64_t)row * dv + col] = S[e];
    }
  }
}

// Many rows of head sizes in whole fours up to 128, aligned: a warp takes four rows (token, head) and has all their loads in flight before the first sum
// (8 sequences of 700..1024 tokens, 16 heads x 128: 34 us after the recurrence with a row a warp, 26 us this way).
__global__ void __launch_bounds__(128) gated_head_norm_vec_kernel(const float* __restrict__ o, const void* __restrict__ w, int dtw,
                                                                  const void* __restrict__ gate, int64_t ldg, int dtg, void* __restrict__ out, int dto,
                                                                  int64_t rows, int H, int dv, float eps, int sigmoid) {
  constexpr int U = 4;
  const uint32_t r0 = (blockIdx.x * 4 + (threadIdx.x >> 5)) * U;
  const int lane = threadIdx.x & 31, c = lane * 4;
  rb::pdl_trigger();
  rb::pdl_wait();
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 x[U], g[U];
#pragma unroll
  for (int i = 0; i < U; ++i) x[i] = r0 + i < rows && c < dv ? *reinterpret_cast<const float4*>(o + (int64_t)(r0 + i) * dv + c) : zero;
#pragma unroll
  for (int i = 0; i < U; ++i) g[i] = r0 + i < rows && c < dv ? rb::ld4_any(gate, dtg, (r0 + i) / (uint32_t)H * ldg + (int)((r0 + i) % (uint32_t)H) * dv + c) : zero;
  const float4 ww = c < dv ? rb::ld4_any(w, dtw, c) : zero;
  auto act = [&](float z) { return (sigmoid ? 1.f : z) / (1.f + expf(-z)); };
#pragma unroll
  for (int i = 0; i < U; ++i) {
    const float4 v = x[i], z = g[i];
    const float rs = 1.f / sqrtf(rb::warp_sum((v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w)) / (float)dv + eps);
    if (r0 + i < rows && c < dv)
      rb::st4_any(out, dto, (int64_t)(r0 + i) * dv + c, make_float4(v.x * rs * ww.x * act(z.x), v.y * rs * ww.y * act(z.y), v.z * rs * ww.z * act(z.z),
                                                                    v.w * rs * ww.w * act(z.w)));
  }
}

// one warp per (token, head), `vec`: four elements per access (sizes and alignment allow it).  With few rows, or more than 128 columns, as fast as or
// faster than rows held in registers (131072 rows x 256 / 512: 74 / 119 us against 76 / 157)
__global__ void __launch_bounds__(128) gated_head_norm_kernel(const float* __restrict__ o, const void* __restrict__ w, int dtw,
                                                              const void* __restrict__ gate, int64_t ldg, int dtg, void* __restrict__ out, int dto,
                                                              int64_t rows, int H, int dv, float eps, int sigmoid, int vec) {
  const int64_t r = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  rb::pdl_trigger();
  rb::pdl_wait();
  if (r >= rows) return;
  const int lane = threadIdx.x & 31;
  const int64_t t = r / H;
  const int h = (int)(r % H);
  const float* x = o + r * dv;
  auto act = [&](float g) { return (sigmoid ? 1.f : g) / (1.f + expf(-g)); };
  float ss = 0.f;
  if (vec) {
    for (int c = lane * 4; c < dv; c += 128) { const float4 v = *reinterpret_cast<const float4*>(x + c); ss += (v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w); }
    ss = rb::warp_sum(ss);
    const float rs = 1.f / sqrtf(ss / (float)dv + eps);
    for (int c = lane * 4; c < dv; c += 128) {
      const float4 v = *reinterpret_cast<const float4*>(x + c), g = rb::ld4_any(gate, dtg, t * ldg + h * dv + c), ww = rb::ld4_any(w, dtw, c);
      rb::st4_any(out, dto, r * dv + c, make_float4(v.x * rs * ww.x * act(g.x), v.y * rs * ww.y * act(g.y), v.z * rs * ww.z * act(g.z),
                                                    v.w * rs * ww.w * act(g.w)));
    }
    return;
  }
  for (int c = lane; c < dv; c += 32) ss += x[c] * x[c];
  ss = rb::warp_sum(ss);
  const float rs = 1.f / sqrtf(ss / (float)dv + eps);
  for (int c = lane; c < dv; c += 32)
    st_any(out, dto, r * dv + c, x[c] * rs * ld_any(w, dtw, c) * act(ld_any(gate, dtg, t * ldg + h * dv + c)));
}

}  // namespace

// blog [T, >= H] / alog [T, >= N]: views with row strides ldb / lda in proj's type; N = H (a decay per head) or H * d (per state row)
extern "C" int rb_delta_prepare(const void* proj, int64_t ld, int dt, const void* conv_w, const void* blog, int64_t ldb, const void* alog, int64_t lda,
                                int N, const void* A_log, const void* dt_bias, float* u, const int* pos, float* conv_state, const int* tok_slot,
                                const int* remain, const int* slots, int64_t T, int H, int G, int d, int dv, int taps, float unit_eps, cudaStream_t s) {
  if (T == 0) return 0;
  if (taps < 1 || taps > kMaxTaps || (N != H && N != H * d)) return -1;
  const GateParams gp{blog, ldb, alog, lda, A_log, dt_bias, N};
  const int units = 2 * G + H + 1 + (N == H ? 0 : H);
  if (pos != nullptr && T >= 64 && d <= 2 * kPThreads && dv <= 2 * kPThreads) {
    // four channels a lane: whole fours of channels, rows of proj and u on their boundaries
    if (d <= 128 && dv <= 128 && d % 4 == 0 && dv % 4 == 0 && ld % 4 == 0 && (H + N) % 4 == 0 && T <= 65535ll * kPThreads &&
        ((reinterpret_cast<uintptr_t>(proj) | reinterpret_cast<uintptr_t>(u)) & 15) == 0) {
      // 32 tokens a warp share their taps and a halo of taps - 1 rows; with fewer than 16 such warps an SM, one tile a warp (1 sequence of 900 tokens, with the
      // recurrence and the norm, 351 us against 360; 8 of 20 .. 40 tokens 37 against 52)
      const int walk = T * units >= (int64_t)rb::kNumSMs * 16 * 32 ? 32 : kTile, per_cta = kPThreads / 32 * walk;
      const dim3 grid(units, (unsigned)((T + per_cta - 1) / per_cta));
      auto go = [&](auto kern) { kern<<<grid, kPThreads, 0, s>>>(proj, ld, dt, conv_w, gp, u, pos, conv_state, tok_slot, remain, T, H, G, d, dv, taps, unit_eps); };
#define RB_GO(T4)                                                                \
  if (walk == 32 && taps <= 4) go(delta_prepare_warp_kernel<T4, 4, 32>);         \
  else if (walk == 32) go(delta_prepare_warp_kernel<T4, kMaxTaps, 32>);          \
  else if (taps <= 4) go(delta_prepare_warp_kernel<T4, 4, kTile>);               \
  else go(delta_prepare_warp_kernel<T4, kMaxTaps, kTile>)
      if (dt == 0) { RB_GO(float); } else if (dt == 1) { RB_GO(__nv_bfloat16); } else { RB_GO(__half); }
#undef RB_GO
      return 0;
    }
    dim3 grid((unsigned)((T + kPT - 1) / kPT), units);
    if (d <= kPThreads && dv <= kPThreads)
      delta_prepare_tiled_kernel<1><<<grid, kPThreads, 0, s>>>(proj, ld, dt, conv_w, gp, u, pos, conv_state, tok_slot, remain, T, H, G, d, dv, taps,
                                                               unit_eps);
    else
      delta_prepare_tiled_kernel<2><<<grid, kPThreads, 0, s>>>(proj, ld, dt, conv_w, gp, u, pos, conv_state, tok_slot, remain, T, H, G, d, dv, taps,
                                                               unit_eps);
    return 0;
  }
  const size_t smem = sizeof(float) * (size_t)(d > dv ? d : dv);
  if (smem > 48 * 1024) return -2;
  if (rb::launch_pdl(delta_prepare_kernel, dim3((unsigned)T, units), dim3(128), smem, s, proj, ld, dt, conv_w, gp, u, pos, conv_state, tok_slot, remain,
                     slots, H, G, d, dv, taps, unit_eps) != cudaSuccess)
    return -3;
  return 0;
}

template <int LPC, int NC, bool CHAN>
static int launch_delta_rule(const ScanParams& p, int n_seqs, cudaStream_t s) {
  constexpr int ncol = kScanThreads / LPC * NC;
  constexpr size_t smem = 2 * sizeof(float) * ((size_t)(CHAN ? 3 : 2) * kTok * 16 * LPC + (size_t)kTok * ncol + 2 * kTok);   // two staging buffers
  auto kern = delta_rule_kernel<LPC, NC, CHAN>;
  if (smem > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -4;
  return rb::launch_pdl(kern, dim3(n_seqs, p.H, RB_CEIL_DIV(p.dv, ncol)), dim3(kScanThreads), smem, s, p) == cudaSuccess ? 0 : -3;
}

template <int LPC, int EPL, bool CHAN>
static int launch_delta_column(const ScanParams& p, int n_seqs, cudaStream_t s) {
  constexpr int ncol = kScanThreads / LPC;
  constexpr size_t smem = 2 * sizeof(float) * ((size_t)(CHAN ? 3 : 2) * kTok * EPL * LPC + (size_t)kTok * ncol + 2 * kTok);   // two staging buffers
  auto kern = delta_column_kernel<LPC, EPL, CHAN>;
  if (smem > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -4;
  return rb::launch_pdl(kern, dim3(n_seqs, p.H, RB_CEIL_DIV(p.dv, ncol)), dim3(kScanThreads), smem, s, p) == cudaSuccess ? 0 : -3;
}

// channel: u rows hold a decay per state row (H * d numbers) instead of one per head
extern "C" int rb_delta_rule(const float* u, float* o, const int* cu, float* s_state, const int* slots, int n_seqs, int H, int G, int d, int dv,
                             int step, int channel, cudaStream_t s) {
  if (n_seqs == 0) return 0;
  if (d > 512 || H % G) return -1;
  ScanParams p{u, o, cu, s_state, slots, H, G, d, dv, step, dv % 4 == 0 && ((uintptr_t)s_state & 15) == 0};
  const bool many = (int64_t)n_seqs * H * RB_CEIL_DIV(dv, 64) >= rb::kNumSMs;
  if (step || (d <= 64 && !(d <= 32 && many))) {       // (lanes per column, state rows per lane)
#define RB_L(LPC, EPL) return channel ? launch_delta_column<LPC, EPL, true>(p, n_seqs, s) : launch_delta_column<LPC, EPL, false>(p, n_seqs, s)
    if (d <= 32) { RB_L(1, 32); }
    if (d <= 64) { RB_L(2, 32); }
    if (d <= 128) { RB_L(2, 64); }
    if (d <= 256) { RB_L(4, 64); }
    RB_L(8, 64);
#undef RB_L
  }
  // (lanes per group, columns per group): 16 LPC state rows; 64 columns a CTA up to head size 128
#define RB_L(LPC, NC) return channel ? launch_delta_rule<LPC, NC, true>(p, n_seqs, s) : launch_delta_rule<LPC, NC, false>(p, n_seqs, s)
  if (d <= 32) { RB_L(2, 1); }
  if (d <= 128) { RB_L(8, 4); }
  if (d <= 256) { RB_L(16, 4); }
  RB_L(32, 4);
#undef RB_L
}

extern "C" int rb_gated_head_norm(const float* o, const void* w, int dtw, const void* gate, int64_t ldg, int dtg, void* out, int dto, int64_t T, int H,
                                  int dv, float eps, int sigmoid, cudaStream_t s) {
  const int64_t rows = T * H;
  if (rows == 0) return 0;
  const bool vec = dv % 4 == 0 && ldg % 4 == 0 && (((uintptr_t)o | (uintptr_t)w | (uintptr_t)gate | (uintptr_t)out) & 15) == 0;
  if (vec && dv <= 128 && rows >= rb::kNumSMs * 64 && rows < (1ll << 31))        // fewer rows: a row a warp keeps more SMs busy
    return rb::launch_pdl(gated_head_norm_vec_kernel, dim3((unsigned)((rows + 15) / 16)), dim3(128), 0, s, o, w, dtw, gate, ldg, dtg, out, dto, rows, H, dv,
                          eps, sigmoid) == cudaSuccess ? 0 : -3;
  return rb::launch_pdl(gated_head_norm_kernel, dim3((unsigned)((rows + 3) / 4)), dim3(128), 0, s, o, w, dtw, gate, ldg, dtg, out, dto, rows, H, dv,
                        eps, sigmoid, (int)vec) == cudaSuccess ? 0 : -3;
}

// Single-token decode attention for sm_100a: fused RoPE + in-place KV append + split-KV online softmax.
//
// One CTA of four warps per (sequence, kv head, kv split); the new token's q/k/v come from the fused QKV projection output, are rotated
// once per CTA, k/v are appended to the dense cache in place, and the CTA streams its slice of the cache once (this op is pure HBM
// bandwidth: 2*S*hd*2 bytes per (sequence, kv head)).  GQA groups (REP query heads per kv head) share every byte.
//
// A warp takes 16 cache rows a step through a ring of its own in shared memory (TMA, so that about 190 KB an SM are on their way
// whatever the arithmetic does, and the load / store unit stays free) and multiplies them on the tensor cores: scores as K [16 keys x hd]
// times q [hd x 8 columns], sums as V^T [hd x 16 keys] times P [16 keys x 8 columns].  Queries and weights are fp32 values and stay so:
// each is the sum of three 16-bit parts (24 bits of a mantissa), and the parts are columns of the same product, (head, part) pairs side by
// side.  A group of one head fills three columns of eight, of two heads six, of four two products, of eight three.  On CUDA cores the same
// step was 3 .. 8 times as many instructions (dot products, butterflies over 16 lanes, broadcasts of the weights), and the SM ran out of
// issue slots and latency before the memory did.
// Measured (B200, room 640, lengths 128 .. 639, no two passes on the same cache; before: CUDA cores, loads into registers, a second kernel to
// merge splits): 128 x 32 heads 145 -> 121 us (6.5 TB/s; reading the same rows and doing nothing takes 113), 16 x 32 heads 27.1 -> 20.6 (16.0 of
// it the kernel), 128 x 8 groups of four heads 95.6 -> 40.6, one group of eight heads a sequence, 20 x 1300 .. 3900, 43.3 -> 17.4.
// A range that has too few (sequence, kv head) pairs to fill the GPU is split over a cluster of 2 .. 8 CTAs, which merge through
// distributed shared memory: no partial sums in global memory and no second kernel.  Infinities and NaN among the cached rows mean what they mean in a plain
// sum (a score of minus infinity: a weight of 0): a warp whose sums are not finite takes its rows again on CUDA cores.  The tensor core's accumulators cut
// off instead of rounding: 1e-6 of the sum over 4000 rows of values of one sign, a hundredth of what rounding the result to 16 bits does.
// Replaces flash_attn_with_kvcache (reference: modules/attn.py:238-251).
#include "attn_common.cuh"

#include <atomic>
#include <type_traits>

namespace {

constexpr int kWarps = 4;
constexpr int kDecThreads = kWarps * 32;
constexpr int kStep = 16;      // cache rows of a warp's step
// CTAs an SM by the query heads of a group (the parts of their queries fill the registers) and the slots of a warp's ring, 16 rows of keys
// or of values each: 150 .. 200 KB an SM
constexpr int ctas_of(int rep) { return rep <= 4 ? 4 : 3; }
constexpr int slots_of(int hd) { return 12288 / (kStep * hd * 2); }
constexpr size_t smem_of(int hd) { return (size_t)kWarps * slots_of(hd) * kStep * hd * 2; }
constexpr int kMaxSplits = 8;  // CTAs of a portable cluster

struct DecodeParams {
  const void* qkv;      // [B, (nq + 2 nkv) * hd]
  void* k_cache;        // logical [B, S, nkv, hd] with arbitrary (b, s, h) strides, unit stride on hd
  void* v_cache;
  const int* cache_lens;  // [B] tokens already cached = position of the new token
  void* out;            // [B, nq * hd]
  const float* cos;     // [max_pos, rot/2] or nullptr
  const float* sin;
  int64_t qkv_stride;
  int64_t kb, ks, kh;   // cache strides in elements
  int64_t vb, vs, vh;
  int B, nq, nkv, S_max, splits, rot_dim, interleaved;
  float scale;
  int* status;          // rb_attn_status()
};

template <typename T> RB_DEVICE void load8(const T* p, float* f) {
  rb::Pack<T, 8> v = *reinterpret_cast<const rb::Pack<T, 8>*>(p);
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = rb::to_f(v.v[i]);
}
template <typename T> RB_DEVICE float2 unpack2(uint32_t r) {
  const T* v = reinterpret_cast<const T*>(&r);
  return make_float2(rb::to_f(v[0]), rb::to_f(v[1]));
}
// Part 0 .. 2 of a pair of fp32 values: their sum is the value to 24 bits.
template <typename T> RB_DEVICE void split2(float a, float b, uint32_t (&part)[3]) {
#pragma unroll
  for (int f = 0; f < 3; ++f) {
    part[f] = pack2<T>(a, b);
    const float2 x = unpack2<T>(part[f]);
    a -= x.x;
    b -= x.y;
  }
}
template <typename T> RB_DEVICE void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, __half>::value)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <bool kTrans> RB_DEVICE void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  if constexpr (kTrans)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <typename T> RB_DEVICE void store8(T* p, const float* f) {
  rb::Pack<T, 8> v;
#pragma unroll
  for (int i = 0; i < 8; ++i) v.v[i] = rb::from_f<T>(f[i]);
  *reinterpret_cast<rb::Pack<T, 8>*>(p) = v;
}

// The cosines and sines of the 8 elements a lane holds of a head (4 pairs if interleaved), read ahead of their use.
struct Angles { float c[8], s[8]; };
RB_DEVICE void load_angles(Angles& t, int sub, const float* cos, const float* sin, int pos, int rot_dim, int interleaved) {
  const int half = rot_dim / 2, d0 = sub * 8;
  if (d0 >= rot_dim) return;
  const int64_t at = (int64_t)pos * half + (interleaved ? d0 / 2 : (d0 < half ? d0 : d0 - half));
  const int n = interleaved ? 4 : 8;
  if (half % 4 == 0 && (reinterpret_cast<uintptr_t>(cos) & 15) == 0 && (reinterpret_cast<uintptr_t>(sin) & 15) == 0 && at % 4 == 0) {
#pragma unroll
    for (int i = 0; i < 8; i += 4)
      if (i < n) {
        const float4 c = *reinterpret_cast<const float4*>(cos + at + i), s = *reinterpret_cast<const float4*>(sin + at + i);
        t.c[i] = c.x; t.c[i + 1] = c.y; t.c[i + 2] = c.z; t.c[i + 3] = c.w;
        t.s[i] = s.x; t.s[i + 1] = s.y; t.s[i + 2] = s.z; t.s[i + 3] = s.w;
      }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < n) { t.c[i] = cos[at + i]; t.s[i] = sin[at + i]; }
  }
}

// Rotate the 8 elements this lane holds of one head.
template <int HD>
RB_DEVICE void rope8(float* x, int sub, const Angles& t, int rot_dim, int interleaved) {
  constexpr int LPR = HD / 8;
  const int half = rot_dim / 2;
  const int d0 = sub * 8;
  if (interleaved) {
    if (d0 < rot_dim) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float a = x[2 * i], b = x[2 * i + 1];
        x[2 * i] = a * t.c[i] - b * t.s[i];
        x[2 * i + 1] = b * t.c[i] + a * t.s[i];
      }
    }
  } else {
    // partner element lives (half) dims away => (half/8) lanes away inside the row's lane group
    const int lane_off = half / 8;
    const bool first = d0 < half;
    const bool active = d0 < rot_dim;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float up = __shfl_down_sync(0xffffffffu, x[i], lane_off, LPR);
      const float dn = __shfl_up_sync(0xffffffffu, x[i], lane_off, LPR);
      if (active) x[i] = first ? (x[i] * t.c[i] - up * t.s[i]) : (x[i] * t.c[i] + dn * t.s[i]);
    }
  }
}

template <typename T, int HD, int REP>
__global__ void __launch_bounds__(kDecThreads, ctas_of(REP)) decode_attn_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                                                                                DecodeParams p) {
  constexpr int LPR = HD / 8;                      // 16-byte pieces of a cache row
  constexpr int NS = slots_of(HD), kSlotBytes = kStep * HD * 2;
  constexpr int kPer = REP == 8 ? 1 : (REP == 4 ? 2 : 3);   // parts side by side in the 8 columns of a product
  constexpr int kProd = (3 + kPer - 1) / kPer;               // products a tile
  extern __shared__ __align__(1024) unsigned char ring[];    // [warp][NS][hd / 64][16 rows][64], 128-byte swizzle
  __shared__ __align__(8) uint64_t bar[kWarps][NS];
  __shared__ uint32_t dead_flag;
  __shared__ __align__(16) float sq[REP][HD], sk[HD], sv[HD];  // the new token, rotated, fp32 (queries: scaled to base-2 units)
  __shared__ __align__(16) T sparts[4][REP][HD + 8];   // the queries' parts, and zeros (rows four banks apart)
  __shared__ float s_unit[REP];                    // fp16: the power of two that a head's queries were brought into range by, inverted
  __shared__ float sm_m[kWarps + 1][REP], sm_l[kWarps + 1][REP];
  __shared__ float cta_m[REP], cta_l[REP];
  float(*cta_acc)[HD] = sq;                        // (the queries' place once the warps are done)
  const int b = blockIdx.x, hkv = blockIdx.y, split = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;           // row / column pair of a tensor-core fragment
  volatile uint32_t* dead = &dead_flag;
  if (threadIdx.x == 0) *dead = 0;
  if (lane < NS) ptx::mbar_init(ptx::smem_u32(&bar[warp][lane]), 1);
  ptx::fence_barrier_init();
  __syncthreads();
  rb::pdl_trigger();  // successors may start launching (and prefetching weights) while this kernel still waits below
  rb::pdl_wait();
  // ---- new token.  A group of hd / 8 lanes rotates one of the REP queries or the key; its values are asked for ahead of the cache rows:
  // behind 190 KB an SM of them these few lines take microseconds to come.
  const int pos = p.cache_lens[b];   // position of the new token; attends to [0, pos]
  const T* qkv = reinterpret_cast<const T*>(p.qkv) + (int64_t)b * p.qkv_stride;
  constexpr int kGroups = kDecThreads / LPR, kTurns = (REP + 1 + kGroups - 1) / kGroups;
  const int sub = threadIdx.x % LPR;
  float xn[kTurns][8], vn[8];
#pragma unroll
  for (int i = 0; i < kTurns; ++i) {
    const int r = threadIdx.x / LPR + i * kGroups;
    load8(qkv + (int64_t)(r < REP ? hkv * REP + r : p.nq + hkv) * HD + sub * 8, xn[i]);
  }
  if (threadIdx.x < LPR) load8(qkv + (int64_t)(p.nq + p.nkv + hkv) * HD + sub * 8, vn);
  Angles ang;
  if (p.cos) load_angles(ang, sub, p.cos, p.sin, pos, p.rot_dim, p.interleaved);

  // ---- this split's range of *cached* positions [lo, hi) (the new token is handled from registers); its first rows are asked for
  const int per = RB_CEIL_DIV(pos, p.splits);
  const int lo = min(pos, split * per), hi = min(pos, lo + per);
  T* kc = reinterpret_cast<T*>(p.k_cache) + (int64_t)b * p.kb + (int64_t)hkv * p.kh;
  T* vc = reinterpret_cast<T*>(p.v_cache) + (int64_t)b * p.vb + (int64_t)hkv * p.vh;
  const uint32_t base = ptx::smem_u32(ring) + warp * NS * kSlotBytes;
  // item n of the warp's sequence K0, V0, K1, V1 .. goes to slot `slot` (rows past the cache read as zeros)
  auto fetch = [&](int n, int slot) {
    const int row0 = lo + ((n >> 1) * kWarps + warp) * kStep;
    if (row0 < hi && ptx::elect_one()) {
      const uint32_t full = ptx::smem_u32(&bar[warp][slot]);
      ptx::mbar_arrive_expect_tx(full, kSlotBytes);
#pragma unroll
      for (int h = 0; h < HD / 64; ++h)
        asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(
                         base + slot * kSlotBytes + h * (kStep * 128)),
                     "l"(n & 1 ? &vmap : &kmap), "r"(full), "r"(h * 64), "r"(row0), "r"(hkv), "r"(b)
                     : "memory");
    }
  };
#pragma unroll
  for (int n = 0; n < NS; ++n) fetch(n, n);

#pragma unroll
  for (int i = 0; i < kTurns; ++i) {
    const int r = threadIdx.x / LPR + i * kGroups;
    if (p.cos) rope8<HD>(xn[i], sub, ang, p.rot_dim, p.interleaved);
    if (r == REP && split == 0 && pos < p.S_max) store8(kc + (int64_t)pos * p.ks + sub * 8, xn[i]);
    float up = p.scale;
    if constexpr (std::is_same<T, __half>::value) {      // the largest element to 2^14 .. 2^15, so that no part of any leaves fp16's range
      float most = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) most = fmaxf(most, fabsf(xn[i][e] * p.scale));
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
      const int ex = (int)(__float_as_uint(most) >> 23) - 127;
      const bool plain = ex < -100 || ex > 100;          // nothing, or nothing finite, to bring into range
      up = plain ? up : up * __uint_as_float((uint32_t)(127 + 14 - ex) << 23);
      if (r < REP && sub == 0) s_unit[r] = plain ? 1.f : __uint_as_float((uint32_t)(127 - 14 + ex) << 23);
    }
    if (r <= REP) {
      float* to = r < REP ? &sq[r][sub * 8] : &sk[sub * 8];
      const float f = r < REP ? up : 1.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) xn[i][e] *= f;
#pragma unroll
      for (int e = 0; e < 8; e += 4) *reinterpret_cast<float4*>(to + e) = make_float4(xn[i][e], xn[i][e + 1], xn[i][e + 2], xn[i][e + 3]);
    }
    if (r < REP) {
      uint32_t part[4][4] = {};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        uint32_t three[3];
        split2<T>(xn[i][2 * e], xn[i][2 * e + 1], three);
        part[0][e] = three[0]; part[1][e] = three[1]; part[2][e] = three[2];
      }
#pragma unroll
      for (int f = 0; f < 4; ++f) *reinterpret_cast<uint4*>(&sparts[f][r][sub * 8]) = make_uint4(part[f][0], part[f][1], part[f][2], part[f][3]);
    }
  }
  if (threadIdx.x < LPR) {
#pragma unroll
    for (int e = 0; e < 8; e += 4) *reinterpret_cast<float4*>(&sv[sub * 8 + e]) = make_float4(vn[e], vn[e + 1], vn[e + 2], vn[e + 3]);
    if (split == 0 && pos < p.S_max) store8(vc + (int64_t)pos * p.vs + sub * 8, vn);
  }
  __syncthreads();

  // ---- the queries as column operands: column g is (part g / REP, head g % REP) of product 0, and so on
  uint32_t qb[HD / 16][kProd][2];
  const int head = g % REP;
#pragma unroll
  for (int c = 0; c < kProd; ++c) {
    const uint32_t* row = reinterpret_cast<const uint32_t*>(&sparts[min(c * kPer + (REP == 8 ? 0 : g / REP), 3)][head][0]) + t;
#pragma unroll
    for (int j = 0; j < HD / 16; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) qb[j][c][h] = row[8 * j + 4 * h];
  }
  if (warp == 0 && split == p.splits - 1) {      // the new token: one more set of partial sums
#pragma unroll
    for (int r = 0; r < REP; ++r) {
      float s = 0.f;
      for (int d = lane; d < HD; d += 32) s = fmaf(sq[r][d], sk[d], s);
      s = rb::warp_sum(s);
      if (lane == 0) {
        sm_m[kWarps][r] = std::is_same<T, __half>::value ? s * s_unit[r] : s;
        sm_l[kWarps][r] = 1.f;
      }
    }
  }
  const float unit = std::is_same<T, __half>::value ? s_unit[head] : 1.f;

  // fragment addresses inside a slot; ^ ((j & 3) << 5) moves them by 16 columns of hd, a block of 64 columns is 2 KB
  const int krow = lane & 15, vrow = (lane & 7) + ((lane >> 4) << 3);
  const uint32_t kat = krow * 128 + (((lane >> 4) ^ (krow & 7)) << 4), vat = vrow * 128 + ((((lane >> 3) & 1) ^ (vrow & 7)) << 4);
  float o[HD / 16][4];
#pragma unroll
  for (int j = 0; j < HD / 16; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  float m = -INFINITY, l = 0.f;                   // of head `head` (l: over the lane's keys)
  int slot = 0;
  uint32_t turn = 0;                              // parity of the ring's current round
  for (int n = 0, row0 = lo + warp * kStep; row0 < hi; n += 2, row0 += kWarps * kStep) {
    // ---- scores of 16 keys: lane (g, t) gets keys g and g + 8 of columns 2t and 2t + 1
    bounded_wait(ptx::smem_u32(&bar[warp][slot]), turn, dead);
    float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
    const uint32_t ka = base + slot * kSlotBytes + kat;
#pragma unroll
    for (int j = 0; j < HD / 16; ++j) {
      uint32_t a[4];
      ldsm4<false>(a, (ka ^ ((j & 3) << 5)) + (j >> 2) * (kStep * 128));
#pragma unroll
      for (int c = 0; c < kProd; ++c) mma16816<T>((j + c) & 1 ? c1 : c0, a, qb[j][c][0], qb[j][c][1]);
    }
    __syncwarp();
    fetch(n + NS, slot);
    if (++slot == NS) { slot = 0; turn ^= 1; }
    // ---- the parts of a head added up, then lane (g, t) takes the keys 2t, 2t + 1, 2t + 8, 2t + 9 of head g % REP
    float s[4];
    {
      float x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = c0[i] + c1[i];
      if constexpr (REP == 1) { x[0] += x[1]; x[2] += x[3]; }
      if constexpr (REP <= 2) {
#pragma unroll
        for (int i = 0; i < 4; i += REP == 1 ? 2 : 1) x[i] += __shfl_xor_sync(0xffffffffu, x[i], 1);
      }
      if constexpr (REP <= 4) {
#pragma unroll
        for (int i = 0; i < 4; i += REP == 1 ? 2 : 1) x[i] += __shfl_xor_sync(0xffffffffu, x[i], 2);
      }
      if constexpr (REP == 8) {
        const int from = 8 * t + (head >> 1);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float even = __shfl_sync(0xffffffffu, x[(i >> 1) * 2], from + (i & 1) * 4), odd = __shfl_sync(0xffffffffu, x[(i >> 1) * 2 + 1], from + (i & 1) * 4);
          s[i] = head & 1 ? odd : even;
        }
      } else {
        // lanes of a row group hold the same sums: each offers one head (t & 1, or for four heads 2 (t & 1) + (t >> 1))
        const bool second = REP == 2 ? t & 1 : (REP == 4 ? t >> 1 : false);
        const float lo8 = second ? x[1] : x[0], hi8 = second ? x[3] : x[2];
        const int from = 8 * t + (REP == 4 ? (head >> 1) | ((head & 1) << 1) : head);
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] = __shfl_sync(0xffffffffu, i < 2 ? lo8 : hi8, from + (i & 1) * 4);
      }
      if constexpr (std::is_same<T, __half>::value) {
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] *= unit;
      }
    }
    if (row0 + kStep > hi) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (row0 + 2 * t + (i & 1) + (i >> 1) * 8 >= hi) s[i] = -INFINITY;
    }
    // ---- running softmax; the accumulators are corrected only where a maximum moved
    float mx = fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2)), m);
    const float zero = mx == -INFINITY ? 0.f : mx;
    if (__any_sync(0xffffffffu, mx != m)) {
      const float corr = exp2f(m - zero);
      l *= corr;
      const float ce = __shfl_sync(0xffffffffu, corr, 8 * t), co = __shfl_sync(0xffffffffu, corr, 8 * t + 4);   // of columns 2t, 2t + 1
#pragma unroll
      for (int j = 0; j < HD / 16; ++j) { o[j][0] *= ce; o[j][1] *= co; o[j][2] *= ce; o[j][3] *= co; }
      m = mx;
    }
    float w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = exp2f(s[i] - zero);
    l += (w[0] + w[1]) + (w[2] + w[3]);
    uint32_t pb[kProd][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      constexpr float kUp = std::is_same<T, __half>::value ? 32768.f : 1.f;    // fp16: small weights keep their bits
      uint32_t part[3];
      split2<T>(w[2 * h] * kUp, w[2 * h + 1] * kUp, part);
#pragma unroll
      for (int c = 0; c < kProd; ++c) {
        const int f = c * kPer + (REP == 8 ? 0 : g / REP);
        pb[c][h] = f == 0 ? part[0] : (f == 1 ? part[1] : (f == 2 ? part[2] : 0u));
      }
    }
    // ---- sums: V^T times the weights' parts
    bounded_wait(ptx::smem_u32(&bar[warp][slot]), turn, dead);
    if (row0 + kStep > hi) {                      // rows that nobody has written yet may hold anything
      for (int i = lane; i < (row0 + kStep - hi) * LPR; i += 32) {
        const int row = kStep - 1 - i / LPR, piece = i % LPR;
        st_shared_v4(base + slot * kSlotBytes + (piece >> 3) * (kStep * 128) + row * 128 + ((piece & 7) << 4), 0, 0, 0, 0);
      }
      __syncwarp();
    }
    const uint32_t va = base + slot * kSlotBytes + vat;
#pragma unroll
    for (int j = 0; j < HD / 16; ++j) {
      uint32_t a[4];
      ldsm4<true>(a, (va ^ ((j & 3) << 5)) + (j >> 2) * (kStep * 128));
#pragma unroll
      for (int c = 0; c < kProd; ++c) mma16816<T>(o[j], a, pb[c][0], pb[c][1]);
    }
    __syncwarp();
    fetch(n + 1 + NS, slot);
    if (++slot == NS) { slot = 0; turn ^= 1; }
  }
  __syncwarp();

  // ---- merge the warps, then the CTAs of the cluster.  A warp's sums take the place of its ring.
  static_assert(NS * kSlotBytes >= REP * HD * 4, "");
  float* mysum = reinterpret_cast<float*>(ring + warp * NS * kSlotBytes);
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  float finite = l * 0.f;                          // 0, or NaN
#pragma unroll
  for (int j = 0; j < HD / 16; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) finite = fmaf(o[j][i], 0.f, finite);
  if (__any_sync(0xffffffffu, finite != 0.f)) {
    // An infinity or a NaN among the keys or values: in a product it meets the zeros beside the parts, and parts of both signs, and what a plain sum
    // makes of it (a weight of 0, an infinite output) is lost.  The warp goes over its rows again, a row at a time in fp32.
#pragma unroll 1
    for (int r = 0; r < REP; ++r) {
      float mr = -INFINITY, lr = 0.f, acc[HD / 32] = {};
#pragma unroll 1
      for (int row0 = lo + warp * kStep; row0 < hi; row0 += kWarps * kStep)
#pragma unroll 1
        for (int row = row0; row < min(row0 + kStep, hi); ++row) {
          float s = 0.f;
#pragma unroll
          for (int e = 0; e < HD / 32; ++e) s = fmaf(sq[r][e * 32 + lane], rb::to_f(kc[(int64_t)row * p.ks + e * 32 + lane]), s);
          s = rb::warp_sum(s);
          if constexpr (std::is_same<T, __half>::value) s *= s_unit[r];
          const float mx = fmaxf(mr, s), zero = mx == -INFINITY ? 0.f : mx, corr = exp2f(mr - zero), w = exp2f(s - zero);
          mr = mx;
          lr = fmaf(lr, corr, w);
#pragma unroll
          for (int e = 0; e < HD / 32; ++e) acc[e] = fmaf(acc[e], corr, w * rb::to_f(vc[(int64_t)row * p.vs + e * 32 + lane]));
        }
      if (lane == 0) { sm_m[warp][r] = mr; sm_l[warp][r] = lr; }
#pragma unroll
      for (int e = 0; e < HD / 32; ++e) mysum[r * HD + e * 32 + lane] = acc[e];
    }
  } else {
    if (g < REP && t == 0) { sm_m[warp][head] = m; sm_l[warp][head] = l; }
#pragma unroll
    for (int j = 0; j < HD / 16; ++j) {
      constexpr float kDown = std::is_same<T, __half>::value ? 1.f / 32768.f : 1.f;
      float x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = o[j][i] * kDown;
      if constexpr (REP == 1) { x[0] += x[1]; x[2] += x[3]; }
      if constexpr (REP <= 2) {
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] += __shfl_xor_sync(0xffffffffu, x[i], 1);
      }
      if constexpr (REP <= 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] += __shfl_xor_sync(0xffffffffu, x[i], 2);
      }
      const int d = 16 * j + g;
      if constexpr (REP == 1) {
        if (t == 0) { mysum[d] = x[0]; mysum[d + 8] = x[2]; }
      } else if (2 * t < REP) {
        mysum[2 * t * HD + d] = x[0];
        mysum[(2 * t + 1) * HD + d] = x[1];
        mysum[2 * t * HD + d + 8] = x[2];
        mysum[(2 * t + 1) * HD + d + 8] = x[3];
      }
    }
  }
  __syncthreads();
  T* out = reinterpret_cast<T*>(p.out) + (int64_t)b * p.nq * HD + (int64_t)hkv * REP * HD;
  const int sets = split == p.splits - 1 ? kWarps + 1 : kWarps;
  for (int idx = threadIdx.x; idx < REP * HD; idx += kDecThreads) {
    const int r = idx / HD, d = idx % HD;
    float mg = -INFINITY;
    for (int w = 0; w < sets; ++w) mg = fmaxf(mg, sm_m[w][r]);
    float lg = 0.f, ag = 0.f;
#pragma unroll
    for (int w = 0; w <= kWarps; ++w) {
      if (w == sets) break;
      const float c = (sm_m[w][r] == -INFINITY) ? 0.f : exp2f(sm_m[w][r] - mg);
      lg += sm_l[w][r] * c;
      ag += (w < kWarps ? reinterpret_cast<const float*>(ring + w * NS * kSlotBytes)[idx] : sv[d]) * c;
    }
    if (p.splits == 1) {
      out[idx] = rb::from_f<T>(lg > 0.f ? ag / lg : 0.f);
    } else {
      cta_acc[r][d] = ag;
      if (d == 0) { cta_m[r] = mg; cta_l[r] = lg; }
    }
  }
  rb::report_given_up(dead, p.status);
  if (p.splits == 1) return;
  ptx::cluster_sync();
  // the cluster is (1, 1, splits): CTA `split` of it finishes its share of the outputs from everybody's sums
  auto peer = [](const float* x, int cta) {
    uint32_t a;
    float v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(ptx::smem_u32(x)), "r"(cta));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
  };
  for (int idx = split * kDecThreads + threadIdx.x; idx < REP * HD; idx += p.splits * kDecThreads) {
    const int r = idx / HD, d = idx % HD;
    float mg = -INFINITY;
    for (int c = 0; c < p.splits; ++c) mg = fmaxf(mg, peer(&cta_m[r], c));
    float lg = 0.f, ag = 0.f;
    for (int c = 0; c < p.splits; ++c) {
      const float mc = peer(&cta_m[r], c), w = mc == -INFINITY ? 0.f : exp2f(mc - mg);
      lg += peer(&cta_l[r], c) * w;
      ag += peer(&cta_acc[r][d], c) * w;
    }
    out[idx] = rb::from_f<T>(lg > 0.f ? ag / lg : 0.f);
  }
  ptx::cluster_sync();  // nobody leaves while its sums are being read
}

template <typename T, int HD, int REP>
int launch_one(const CUtensorMap& kmap, const CUtensorMap& vmap, const DecodeParams& p, cudaStream_t s) {
  static std::atomic<uint64_t> opted_in{0};          // the attribute is the kernel's on one device: a bit per device
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -3;
  if (dev >= 64 || !(opted_in.load(std::memory_order_relaxed) >> dev & 1)) {
    if (cudaFuncSetAttribute(decode_attn_kernel<T, HD, REP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_of(HD)) != cudaSuccess) return -3;
    if (dev < 64) opted_in.fetch_or(uint64_t(1) << dev, std::memory_order_relaxed);
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(p.B, p.nkv, p.splits);
  cfg.blockDim = dim3(kDecThreads);
  cfg.dynamicSmemBytes = smem_of(HD);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (p.splits > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = p.splits;
  }
  if (rb::pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, decode_attn_kernel<T, HD, REP>, kmap, vmap, p) == cudaSuccess ? 0 : -3;
}

// [B, S, nkv, hd] with any strides as boxes of 16 rows x 64 columns of one head.
bool cache_map(CUtensorMap* m, const void* ptr, int is_bf16, int B, int S, int nkv, int hd, int64_t sb, int64_t ss, int64_t sh) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return false;
  static thread_local bool ctx_ready = false;     // (as in make_tmap: the driver call needs this thread's context bound)
  if (!ctx_ready) { cudaFree(nullptr); ctx_ready = true; }
  cuuint64_t dims[4] = {(cuuint64_t)hd, (cuuint64_t)S, (cuuint64_t)nkv, (cuuint64_t)B};
  // (the stride of a dimension of one is never used, and may be anything)
  cuuint64_t strides[3] = {(cuuint64_t)(S > 1 ? ss : hd) * 2, (cuuint64_t)(nkv > 1 ? sh : hd) * 2, (cuuint64_t)(B > 1 ? sb : hd) * 2};
  cuuint32_t box[4] = {64, (cuuint32_t)kStep, 1, 1}, estr[4] = {1, 1, 1, 1};
  return fn(m, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename T, int HD>
int launch_decode(const DecodeParams& p, cudaStream_t s) {
  CUtensorMap kmap, vmap;
  constexpr int bf = std::is_same<T, __nv_bfloat16>::value;
  if (!cache_map(&kmap, p.k_cache, bf, p.B, p.S_max, p.nkv, HD, p.kb, p.ks, p.kh) || !cache_map(&vmap, p.v_cache, bf, p.B, p.S_max, p.nkv, HD, p.vb, p.vs, p.vh)) return -4;
  switch (p.nq / p.nkv) {
    case 1: return launch_one<T, HD, 1>(kmap, vmap, p, s);
    case 2: return launch_one<T, HD, 2>(kmap, vmap, p, s);
    case 4: return launch_one<T, HD, 4>(kmap, vmap, p, s);
    case 8: return launch_one<T, HD, 8>(kmap, vmap, p, s);
    default: return -1;
  }
}

}  // namespace

extern "C" int rb_decode_attention(const void* qkv, void* k_cache, void* v_cache, const int* cache_lens, void* out, const float* cos,
                                   const float* sin, int64_t qkv_stride, int64_t kb, int64_t ks, int64_t kh, int64_t vb, int64_t vs, int64_t vh,
                                   int B, int nq, int nkv, int hd, int S_max, int rot_dim, int interleaved, float scale, int dt, cudaStream_t s) {
  if (B == 0) return 0;
  // CTAs a (sequence, kv head) pair: doubled as long as all of them still fit at once (ctas_of) and a CTA keeps at least two steps (2 x 64 rows)
  // of a full cache.  A second round of CTAs costs more than shorter ones give: 16 x 32 heads (512 CTAs for 592 places) 20.8 us whole, 25.1 in
  // halves; 32 heads of one sequence of 3900 tokens 46.7 whole, 28.2 / 21.9 / 15.4 in 2 / 4 / 8; 16 x 8 groups of four heads, up to 1900 tokens,
  // 26.2 whole, 20.4 / 17.4 / 22.8 in 2 / 4 / 8.
  const int rep = nq / nkv, slots = rb::kNumSMs * ctas_of(rep), rows = 2 * kWarps * kStep;
  int splits = 1;
  while (splits < kMaxSplits && (int64_t)B * nkv * splits * 2 <= slots && S_max >= rows * splits * 2) splits *= 2;
  DecodeParams p{qkv, k_cache, v_cache, cache_lens, out, cos, sin, qkv_stride, kb, ks, kh, vb, vs, vh,
                 B, nq, nkv, S_max, splits, rot_dim, interleaved, scale * 1.4426950408889634f, rb_attn_status()};
  if (p.status == nullptr) return -5;
  if (dt == 1 && hd == 128) return launch_decode<__nv_bfloat16, 128>(p, s);
  if (dt == 1 && hd == 64) return launch_decode<__nv_bfloat16, 64>(p, s);
  if (dt == 2 && hd == 128) return launch_decode<__half, 128>(p, s);
  if (dt == 2 && hd == 64) return launch_decode<__half, 64>(p, s);
  return -2;
}
